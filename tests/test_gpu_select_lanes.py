"""With 8 paths a selection lane takes one run of 16 disparities at every size: the volumes'
bytes bound it, and lanes that take more runs read them in smaller pieces."""
import pytest

from tests import gpu_graph, gpu_util as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("disparities,lanes", [(64, 4), (96, 8), (128, 8), (192, 16), (256, 16)])
def test_one_run_a_lane_with_eight_paths(disparities, lanes):
    from nx_stereo_b200 import native

    width, height = 1024, 600  # above and below half a million pixels, where a rule changed lanes
    for h in (height, 200):
        volumes = g.empty(16, g.torch().uint8)  # captured, not run
        out = g.empty((h, width), g.torch().float32)
        launched = gpu_graph.kernels_of(lambda stream: native.call(
            "nxs_select_paths_device_ordered", g.ptr(volumes), width, h, disparities, 8, 1.05, 16,
            g.ptr(out), g.ptr(out), stream))
        assert [f"select_kernelILi{lanes}ELi8ELi16ELi1E" in k.name for k in launched] == [True], \
            launched
