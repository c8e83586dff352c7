"""The quality sums at the edges of their kernel's blocks (8 columns, 128 rows in flight),
against the oracle. Sums of counts and values in f64, rounded to f32 once a column and once in
all: whatever the order of the f64 additions, the two roundings bound the difference from the
oracle's by 2^-23 + 2^-24 of the sum (all terms are positive), below 1e-6."""
import numpy as np
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def native():
    from nx_stereo_b200 import native as n

    n.load()
    return n


@pytest.mark.parametrize("w,h", [(1, 1), (7, 63), (8, 64), (9, 65), (33, 130), (500, 3), (8, 128), (9, 257)])
def test_quality_sums_at_the_edges_of_its_blocks(native, oracle, w, h):
    """Widths and heights around a block, a frame of unmatched pixels, and the disparity moved
    into `previous`."""
    rng = np.random.default_rng(w * 100 + h)
    maps = [np.where(rng.random((h, w)) < 0.3, -1, rng.uniform(0.5, 90, (h, w))).astype(np.float32)
            for _ in range(2)] + [np.full((h, w), -1, np.float32)]
    previous = np.full((h, w), -1, np.float32)
    d_previous, d_sums = g.dev(previous), g.empty(5, g.torch().float32)
    for current in maps:
        want, previous = oracle.quality(current, previous)
        native.call("nxs_quality_device", g.ptr(g.dev(current)), g.ptr(d_previous), w, h,
                    g.ptr(d_sums), g.stream())
        assert np.allclose(g.host(d_sums), want, rtol=1e-6, atol=0)
        assert g.same_bits(g.host(d_previous), current)
