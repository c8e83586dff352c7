"""The path scan in the sweep order (every line of a direction at the same image row, diagonal
lines going on at the other side) against the scan of the ranked lines (tiles mode 0), which the
oracle pins: every disparity count it takes, both path counts, both orders of its warps, widths
and heights that do not fill warps, and a pair higher than wide, whose diagonal lines go around
more than once. The path volumes are compared bit for bit."""
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu

# pairs just above where the sweep begins, by disparity count
CASES = [(1031, 1021, 64, 8), (517, 2049, 64, 8), (131, 8011, 64, 3), (1031, 1021, 64, 3),
         (953, 737, 96, 8), (1021, 517, 128, 8), (4093, 131, 128, 8), (519, 1013, 128, 3),
         (1279, 701, 192, 8), (733, 359, 256, 3), (2047, 2049, 64, 8), (1920, 1079, 192, 8),
         (1163, 907, 256, 8)]


@pytest.mark.parametrize("width,height,disparities,paths", CASES)
def test_the_sweep_writes_the_ranked_lines_volumes(width, height, disparities, paths):
    from nx_stereo_b200 import native

    lib, torch = native.load(), g.torch()
    cells = width * height * disparities
    assert cells >= 64 << 20
    generator = torch.Generator(device="cuda").manual_seed(cells)
    costs = torch.randint(0, 49, (cells,), generator=generator, device="cuda", dtype=torch.uint8)
    costs[:: 1009] = 48
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
