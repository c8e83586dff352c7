"""Selection at every number of runs a lane takes: each path count and disparity count in both
of the matcher's orders, on path volumes that reach the winner's edges (ties, winners at the
first and last disparity and on either side of a run, disparities past the left edge), against
the selection of their u16 sums (one run a lane, held to the oracle by the tests of the steps),
bit for bit; pixel counts around a block's."""
import numpy as np
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu


def _order(span, disparities):
    d = np.arange(disparities)
    if span == 0:
        return d
    half = span // 2
    return (d // span) * span + 4 * ((d % span % half) // 2) + d % 2 + 2 * (d % span // half)


@pytest.mark.parametrize("paths", [3, 8])
@pytest.mark.parametrize("disparities", [64, 80, 96, 128, 192, 256])
def test_selection_of_every_run_count(disparities, paths):
    from nx_stereo_b200 import native

    lib = native.load()
    torch = g.torch()
    rng = np.random.default_rng(disparities * 10 + paths)
    sizes = [(9, 7), (65, 3), (300, 2)]
    if paths == 8 and disparities == 64:
        sizes += [(4096, 128), (4097, 128)]  # where two runs a lane begin with 8 paths
    for width, height in sizes:
        volumes = rng.integers(0, 113, (paths, height, width, disparities)).astype(np.uint8)
        low = rng.integers(0, disparities, (height, width))
        low[:, ::3] = rng.choice([0, 1, 15, 16, 47, 48, disparities - 1], low[:, ::3].shape)
        np.put_along_axis(volumes, np.broadcast_to(low[None, :, :, None], (paths, height, width, 1)),
                          3, axis=3)
        volumes[:, :, 1::4] = 7  # ties everywhere
        sums = volumes.astype(np.uint16).sum(0, dtype=np.uint16)
        want_d, want_k = g.empty((height, width), torch.float32), g.empty((height, width), torch.int32)
        native.call("nxs_select_device", g.ptr(g.dev(sums.view(np.int16))), width, height,
                    disparities, 1.05, g.ptr(want_d), g.ptr(want_k), g.stream())
        for span in (0, 8, 16):
            ordered = np.empty_like(volumes)
            ordered[..., _order(span, disparities)] = volumes
            got_d, got_k = torch.empty_like(want_d), torch.empty_like(want_k)
            native.call("nxs_select_paths_device_ordered", g.ptr(g.dev(ordered)), width, height,
                        disparities, paths, 1.05, span, g.ptr(got_d), g.ptr(got_k), g.stream())
            assert g.same_bits(g.host(got_d), g.host(want_d)), (width, height, span)
            assert (g.host(got_k) == g.host(want_k)).all(), (width, height, span)
