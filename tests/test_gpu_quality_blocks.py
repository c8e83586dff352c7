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


def test_a_captured_call_before_any_other():
    """The first call of a process may be a captured one: its scratch is the graph's."""
    import subprocess
    import sys

    code = """
import numpy as np, torch
from nx_stereo_b200 import native
d = torch.rand((40, 50), device="cuda") * 50
previous, sums = torch.full_like(d, -1.0), torch.empty(5, device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    native.call("nxs_quality_device", d.data_ptr(), previous.data_ptr(), 50, 40,
                sums.data_ptr(), torch.cuda.current_stream().cuda_stream)
graph.replay()
torch.cuda.synchronize()
assert sums[0].item() == 2000 and abs(sums[1].item() / d.sum().item() - 1) < 1e-5
assert torch.equal(previous, d)
"""
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
