"""Which order the path scan takes a pair's lines in, on both sides of each line of the rule
(read from the launch, which does not run), and the sweep order's volumes for the narrowest
and shortest pairs it can be given: lines that go around every 9 steps, warps of lines that no
column fills, fewer rows than a lane keeps in flight. The volumes are those of the ranked lines
(tiles mode 0), which the oracle pins, bit for bit."""
import re

import pytest

from tests import gpu_graph, gpu_util as g

pytestmark = pytest.mark.gpu


def _order(width, height, disparities, paths):
    from nx_stereo_b200 import native

    buffer = g.empty(256, g.torch().uint8)
    (kernel,) = gpu_graph.kernels_of(lambda stream: native.call(
        "nxs_paths_device_ordered", g.ptr(buffer), width, height, disparities, paths, 8, 64, 16,
        g.ptr(buffer), stream))
    if "paths_sweep_kernel" in kernel.name:
        return "sweep"
    # paths_kernel<G, WORDS, FULL, SPAN, SUMS, TILES>
    return "tiles" if re.search(r"paths_kernelI(Li\d+E){2}Lb1ELi16ELb0ELb1EE", kernel.name) else "ranked"


ORDERS = [
    # 8 paths
    (1440, 810, 64, "ranked"), (1600, 900, 64, "ranked"), (1700, 1000, 64, "sweep"),
    (900, 1200, 64, "sweep"), (1200, 900, 64, "ranked"), (3000, 1900, 64, "sweep"),
    (3840, 2160, 64, "tiles"), (990, 700, 96, "ranked"), (1000, 750, 96, "sweep"),
    (3840, 2160, 96, "sweep"), (728, 544, 128, "ranked"), (960, 600, 128, "sweep"),
    (1600, 1000, 128, "sweep"), (1600, 1280, 128, "tiles"), (1920, 1080, 128, "sweep"),
    (1080, 1920, 128, "sweep"), (1280, 1600, 128, "tiles"), (2560, 1440, 128, "tiles"),
    (800, 600, 192, "ranked"), (1280, 720, 192, "sweep"), (2560, 1440, 192, "sweep"),
    (1920, 1080, 160, "sweep"), (1920, 1080, 224, "sweep"), (640, 480, 256, "ranked"),
    (1280, 720, 256, "tiles"), (1400, 800, 256, "tiles"), (1920, 1080, 256, "sweep"),
    (1080, 1920, 256, "tiles"), (2048, 1400, 256, "tiles"),
]
ORDERS_3 = [
    (1920, 1080, 64, "ranked"), (2560, 1920, 64, "ranked"), (3840, 2600, 64, "tiles"),
    (1920, 1080, 96, "ranked"), (2560, 1440, 96, "sweep"), (3840, 2160, 96, "ranked"),
    (1280, 720, 128, "ranked"), (2560, 1440, 128, "sweep"), (3840, 2160, 128, "tiles"),
    (1920, 1080, 192, "ranked"), (900, 600, 256, "ranked"), (1280, 720, 256, "sweep"),
    (2560, 1440, 256, "tiles"),
]


@pytest.mark.parametrize("width,height,disparities,paths,order",
                         [(w, h, d, 8, o) for w, h, d, o in ORDERS] +
                         [(w, h, d, 3, o) for w, h, d, o in ORDERS_3])
def test_the_order_of_a_pairs_lines(width, height, disparities, paths, order):
    assert _order(width, height, disparities, paths) == order


@pytest.mark.parametrize("width,height,disparities,paths", [
    (9, 116509, 64, 8), (13, 80660, 64, 8), (33, 31776, 64, 8), (9, 77673, 96, 8),
    (77673, 9, 96, 8), (9, 58255, 128, 8), (58255, 9, 128, 8), (15, 34953, 128, 8),
    (74899, 7, 128, 8), (9, 116509, 160, 8), (9, 97091, 192, 8), (97091, 9, 192, 8),
    (9, 83221, 224, 8), (9, 407785, 96, 3), (407785, 9, 128, 3), (9, 407785, 128, 3),
    (9, 100126, 256, 3), (100126, 9, 256, 3)])
def test_the_sweep_of_narrow_and_short_pairs(width, height, disparities, paths):
    from nx_stereo_b200 import native

    assert _order(width, height, disparities, paths) == "sweep"
    lib, torch = native.load(), g.torch()
    cells = width * height * disparities
    generator = torch.Generator(device="cuda").manual_seed(cells)
    costs = torch.randint(0, 49, (cells,), generator=generator, device="cuda", dtype=torch.uint8)
    volumes = {}
    for mode in (0, 1):
        volumes[mode] = torch.zeros(paths * cells, device="cuda", dtype=torch.uint8)
        assert lib.nxs_set_path_tiles(mode) == 0
        try:
            native.call("nxs_paths_device_ordered", costs.data_ptr(), width, height, disparities,
                        paths, 5, 79, 16, volumes[mode].data_ptr(), g.stream())
        finally:
            lib.nxs_set_path_tiles(1)
    torch.cuda.synchronize()
    assert torch.equal(volumes[0], volumes[1])
