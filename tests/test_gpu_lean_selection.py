"""The selection that runs beside other pairs' path scans (a grid of a few resident blocks a
SM), with 3 paths at every disparity count: the stream engine's disparities are those of a
pair by itself, bit for bit, also where each resident block takes several pixel blocks; and an
SM holds the blocks that the grid is sized for, whatever the lanes' runs of disparities."""
import json

import numpy as np
import pytest

from tests import gpu_util as g

pytestmark = pytest.mark.gpu

DISPARITIES = [64, 96, 128, 192, 256]


@pytest.fixture(scope="module")
def ctx():
    from nx_stereo_b200 import native

    c = native.Context(0)
    yield c
    c.close()


def _plan(ctx, shapes):
    from nx_stereo_b200 import batch

    return batch.BatchPlan(ctx, shapes, {"engine": 1, "streams": 2})


@pytest.mark.parametrize("paths", [3, 8])
@pytest.mark.parametrize("disparities", DISPARITIES)
def test_lean_selection_with_either_path_count(ctx, disparities, paths):
    """One resident block a SM (148 of them) over 1,300 to 12,000 pixel blocks, and the
    default; a ragged last block in both sizes."""
    from nx_stereo_b200 import native

    lib, torch = native.load(), g.torch()
    shapes = [(w, h, {"disparities": disparities, "paths": paths}) for w, h in ((301, 211), (333, 145))]
    generator = np.random.default_rng(disparities + paths)
    for lean in (1, 8):
        assert lib.nxs_set_lean_select(lean) == 0
        try:
            plan = _plan(ctx, shapes)
            pairs = []
            for k, (w, h, _) in enumerate(shapes):
                left = generator.integers(0, 256, (h, w)).astype(np.uint8)
                right = np.roll(left, -9 - 30 * k, axis=1)
                right[:, ::7] = generator.integers(0, 256, right[:, ::7].shape)
                views = plan.device_views(k)
                views[0].copy_(torch.from_numpy(left))
                views[1].copy_(torch.from_numpy(right))
                pairs.append((left, right))
            plan.launch(stream=g.stream())
            torch.cuda.synchronize()
            got = [plan.device_views(k)[2].cpu().numpy() for k in range(len(shapes))]
            plan.close()
        finally:
            lib.nxs_set_lean_select(8)
        for (left, right), disparity in zip(pairs, got):
            want = ctx.sgm(left, right, disparities=disparities, paths=paths)
            assert g.same_bits(disparity, want), lean


@pytest.mark.parametrize("paths", [3, 8])
def test_an_sm_holds_the_lean_grid(ctx, tmp_path, paths):
    """The registers of the launches, from the profiler's trace: an SM's 65,536 hold the
    default grid's blocks of 128 threads."""
    from torch.profiler import ProfilerActivity, profile

    from nx_stereo_b200 import native

    torch = g.torch()
    plans = [_plan(ctx, [(301, 211, {"disparities": d, "paths": paths})] * 2) for d in DISPARITIES]
    for plan in plans:
        plan.launch(stream=g.stream())
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as trace:
        for plan in plans:
            plan.launch(stream=g.stream())
        torch.cuda.synchronize()
    for plan in plans:
        plan.close()
    trace.export_chrome_trace(str(tmp_path / "trace.json"))
    with open(tmp_path / "trace.json") as file:
        events = json.load(file)["traceEvents"]
    registers = {e["name"]: e["args"]["registers per thread"] for e in events
                 if "select_lean_kernel" in e.get("name", "") and "args" in e}
    assert len(registers) == len(DISPARITIES) - (paths == 8) * 2, registers
    most = 65536 // (native.load().nxs_lean_select() * 128)
    assert all(used <= most for used in registers.values()), registers
