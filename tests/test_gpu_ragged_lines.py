"""Scan lines that do not fill their warps: line counts that are no multiple of a warp's
lines (the last warp follows its last line again, without writing), disparity counts that
do not fill a line's lanes, lines shorter than and just around the ring of costs a lane
keeps in flight, through the path volumes and through the summing scan (where a line
followed twice must add once). Every output is the oracle's, bit for bit."""
import numpy as np
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu

# width x height: the smallest pair, lines of 7..13, 23..25 and 31..33 steps, and rows and
# columns of every remainder by 2, 4 and 8 lines a warp
SIZES = [(9, 7), (13, 8), (23, 12), (24, 25), (33, 31), (50, 13), (97, 30)]


@pytest.fixture(scope="module")
def ctx():
    from nx_stereo_b200 import native

    c = native.Context(0)
    yield c
    c.close()


def _pair(width, height):
    rng = np.random.default_rng(width * 1000 + height)
    left = rng.integers(0, 256, (height, width)).astype(np.uint8)
    right = np.roll(left, -3, axis=1)
    right[:, ::5] = rng.integers(0, 256, right[:, ::5].shape)
    return left, right


@pytest.mark.parametrize("paths", [3, 8])
@pytest.mark.parametrize("disparities", [64, 96, 128, 192, 256])
def test_ragged_lines_match_the_oracle(ctx, oracle, disparities, paths):
    from nx_stereo_b200 import native

    lib = native.load()
    for width, height in SIZES:
        left, right = _pair(width, height)
        want = oracle.sgm(left, right, disparities, paths, p1=5, p2=79, uniqueness=1.1)
        for sums in (0, 1):
            lib.nxs_set_path_sums(sums)
            try:
                got = ctx.sgm(left, right, disparities=disparities, paths=paths, p1=5, p2=79,
                              uniqueness=1.1)
            finally:
                lib.nxs_set_path_sums(0)
            assert g.same_bits(got, want), (width, height, sums)
