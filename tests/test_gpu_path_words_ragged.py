"""4 and 16 words a path lane on lines that do not fill their warps or their lanes and are as
short as the costs kept in flight: the oracle's disparities, bit for bit."""
import numpy as np
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [4, 16])
@pytest.mark.parametrize("disparities", [64, 96, 128, 192, 256])
def test_ragged_lines_with_other_words_a_lane(oracle, disparities, words):
    from nx_stereo_b200 import native

    lib, ctx = native.load(), native.Context(0)
    saved = lib.nxs_path_words(disparities)
    assert lib.nxs_set_path_words(disparities, words) == 0
    try:
        for width, height in [(9, 7), (13, 8), (23, 12), (24, 25), (33, 31), (50, 13), (97, 30)]:
            rng = np.random.default_rng(width * height + disparities)
            left = rng.integers(0, 256, (height, width)).astype(np.uint8)
            right = np.roll(left, -3, axis=1)
            right[:, ::5] = rng.integers(0, 256, right[:, ::5].shape)
            for paths in (3, 8):
                want = oracle.sgm(left, right, disparities, paths, p1=5, p2=79, uniqueness=1.1)
                got = ctx.sgm(left, right, disparities=disparities, paths=paths, p1=5, p2=79,
                              uniqueness=1.1)
                assert g.same_bits(got, want), (width, height, paths)
    finally:
        lib.nxs_set_path_words(disparities, saved)
        ctx.close()
