"""The pool that the quality sums' scratch comes from: kept between calls, given back when a
context on the device is destroyed, made anew for the next call."""
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu


def test_a_destroyed_context_gives_the_small_pool_back():
    from nx_stereo_b200 import native

    torch, ctx = g.torch(), native.Context(0)
    width, height = 50, 40
    disparity = torch.rand((height, width), device="cuda") + 1
    previous, sums = torch.full_like(disparity, -1.0), g.empty(5, torch.float32)

    def call():
        native.call("nxs_quality_device", g.ptr(disparity), g.ptr(previous), width, height,
                    g.ptr(sums), g.stream())
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    kept = call()
    assert call() == kept
    ctx.close()
    assert torch.cuda.mem_get_info()[0] - kept >= 32 << 20
    assert call() == kept and sums[0].item() == width * height
