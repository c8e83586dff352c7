"""The work that users of nx_stereo_b200 have it do, as cases that can be timed.

`listed()` gives the cases, `draw(rng)` more of the same ranges, `prepare(case,
seed)` what a program holds before the call, `run(state)` one pass through the
public entry points, `work(case)` what a pass cannot do without, and
`exact(case, seed)` the pass's results from plain torch in 64 bits (whole-number
steps as whole numbers), where they are determined to that precision.

Kinds of case:
  sgm       NxStereo.sgm/3 on a rectified pair in device memory (Context.sgm_device)
  c2f       sgm_coarse_to_fine/3 on one (Context.sgm_coarse_to_fine_device)
  stages    the stages around the matcher, each by its device entry point
  pipeline  frames in host memory through a CudaSegment that carries nothing
  stream    frames of one camera stream through a CudaSegment that carries state
  batch     a BatchPlan over rectified pairs of mixed sizes, in device memory
"""
import ctypes

import numpy as np
import torch

from nx_stereo_b200 import batch, native, scene, segment, stage

UNIQUENESS = stage.DEFAULT_UNIQUENESS


# ---------------------------------------------------------------- the cases
def _sgm(width, height, disparities, paths=8, p1=8, p2=64, uniqueness=UNIQUENESS):
    return {"kind": "sgm", "width": width, "height": height, "disparities": disparities,
            "paths": paths, "p1": p1, "p2": p2, "uniqueness": uniqueness}


def _c2f(width, height, band=16, paths=8, census="sparse_9x7"):
    return {"kind": "c2f", "width": width, "height": height, "band": band, "paths": paths,
            "census": census}


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # The smallest calls in use: a thumbnail-sized depth estimate, where launches
        # and one wave's latency count.
        named("sgm_320x240_d64", _sgm(320, 240, 64)),
        # A small board's working size with the faster 3-path mode.
        named("sgm_480x270_d64_p3", _sgm(480, 270, 64, paths=3)),
        # An odd crop with a disparity range that does not fill its lanes, and settings
        # of the user's own.
        named("sgm_641x479_d96", _sgm(641, 479, 96, p1=5, p2=79, uniqueness=1.2)),
        # The headline size.
        named("sgm_728x544_d128", _sgm(728, 544, 128)),
        # A 720p camera, the larger stream of the serving workload.
        named("sgm_1280x720_d128", _sgm(1280, 720, 128)),
        # A ragged 720p crop with a near-range search in 3 paths.
        named("sgm_1277x713_d192_p3", _sgm(1277, 713, 192, paths=3)),
        # The largest: full HD at the widest search.
        named("sgm_1920x1080_d256", _sgm(1920, 1080, 256)),
        # The coarse-to-fine search at the headline size.
        named("c2f_728x544_b16", _c2f(728, 544)),
        # A caller with its own matcher that takes the stages around it.
        named("stages_1280x720", {"kind": "stages", "width": 1280, "height": 720}),
        # The full frame-to-depth pipeline as a program drives it: host frames, up to the
        # segment's depth of pairs in flight, every output back on the host.
        named("pipeline_728x544_d128", {"kind": "pipeline", "width": 728, "height": 544,
                                        "disparities": 128, "pairs": 8}),
        # A camera stream of the serving workload: the stages that carry state.
        named("stream_1280x720_d128", {"kind": "stream", "width": 1280, "height": 720,
                                       "disparities": 128, "pairs": 4}),
        # An offline job: a planned batch of mixed sizes and ranges, on the engine the
        # autotuner settles on for such mixes.
        named("batch_16_mixed", {"kind": "batch", "pairs": 16, "mix": 5}),
    ]


def draw(rng):
    def spread(low, high):
        return int(round(low * (high / low) ** rng.random()))

    kind = rng.choices(["sgm", "c2f", "stages", "pipeline", "stream", "batch"],
                       [9, 2, 1, 1, 1, 1])[0]
    width = spread(320, 1920)
    height = max(200, min(1080, int(width * rng.uniform(0.55, 0.78))))
    if kind == "sgm":
        p1 = rng.randint(3, 12)
        return _sgm(width, height, rng.choice([64, 96, 128, 128, 192, 256]),
                    paths=rng.choice([8, 8, 8, 3]), p1=p1, p2=rng.randint(p1 + 20, 79),
                    uniqueness=rng.choice([1.0, UNIQUENESS, 1.2]))
    if kind == "c2f":
        return _c2f(width // 2 * 2, height // 2 * 2, band=rng.choice([8, 16, 16, 32]),
                    paths=rng.choice([8, 8, 3]),
                    census=rng.choice(["sparse_9x7", "dense_9x5", "dense_9x5_blend"]))
    if kind == "stages":
        return {"kind": kind, "width": width, "height": height}
    if kind in ("pipeline", "stream"):
        width = spread(320, 1280)
        return {"kind": kind, "width": width, "height": int(width * rng.uniform(0.55, 0.75)),
                "disparities": rng.choice([64, 128]), "pairs": rng.randint(2, 8)}
    return {"kind": kind, "pairs": rng.randint(4, 16), "mix": rng.randrange(1 << 20)}


def _batch_shapes(case):
    return batch.sample_shapes(case["pairs"], case["mix"])


def work(case):
    """Bytes: each input read and each output written once. Operations: the census's
    comparisons, the costs' XORs and counts, and per path and cell the recurrence's
    three minimums and two sums, then the sum of the paths and the winner's search."""
    def matcher(pixels, cells, paths):
        return pixels * 48 * 2 + cells * (2 + 5 * paths + paths + 2)

    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(6 * w * h for w, h, _ in shapes),
                "flops": sum(matcher(w * h, w * h * s["disparities"], s["paths"])
                             for w, h, s in shapes)}
    px = case["width"] * case["height"]
    if kind == "sgm":
        return {"bytes": 6 * px, "flops": matcher(px, px * case["disparities"], case["paths"])}
    if kind == "c2f":
        return {"bytes": (2 + 4 + 4) * px,
                "flops": matcher(px // 4, px // 4 * 64, case["paths"]) +
                matcher(px, px * case["band"], case["paths"])}
    if kind == "stages":  # both frames, two disparities and the carried maps in; the outputs
        return {"bytes": px * (2 + 2 + 4 + 4 + 8 + 8 + 2 + 4 + 4 + 4) + px // 16 * 12,
                "flops": px * (2 * 60 + 48 * 4 + 10 + 6 + 10)}
    per_pair = 2 * px + 2 * px + 4 * px + 2 * px
    return {"bytes": case["pairs"] * per_pair,
            "flops": case["pairs"] * (matcher(px, px * case["disparities"], 8) +
                                      px * (2 * 30 + 48 * 4 + 12))}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _pair(width, height, gen, nearest):
    """A rectified u8 pair of a textured scene: a slanted background and a few nearer
    rectangles, the left view sampled from the right one at its disparity, both with
    sensor noise; flat and shaded patches among the texture."""
    def uniform(n, low, high):
        return (low + (high - low) * torch.rand(n, generator=gen, device="cuda")).tolist()

    noise = torch.rand((1, 1, height, width + 2 * nearest), generator=gen, device="cuda") * 255
    texture = torch.nn.functional.avg_pool2d(
        torch.nn.functional.pad(noise, (1, 1, 1, 1), mode="replicate"), 3, 1)[0, 0]
    yy = torch.arange(height, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(width + 2 * nearest, device="cuda", dtype=torch.float32)[None, :]
    for u, v, s, g in zip(*(uniform(3, *r) for r in ((0, 1), (0, 1), (0.1, 0.3), (-0.2, 0.2)))):
        box = ((xx >= u * width) & (xx < (u + s) * width) & (yy >= v * height) &
               (yy < (v + s) * height))
        texture = torch.where(box, 0.4 * texture + 0.6 * (128 + g * (xx - u * width)), texture)
    x = torch.arange(width, device="cuda", dtype=torch.float32)[None, :]
    far, slope_x, slope_y = uniform(1, 8, 14) + uniform(2, -4, 4)
    disparity = (far + slope_x * x / width + slope_y * yy / height).clamp(4, 20)
    for u, v, s, d in zip(*(uniform(6, *r) for r in ((0, 0.8), (0, 0.8), (0.1, 0.33),
                                                     (8, nearest - 4)))):
        box = ((x >= u * width) & (x < (u + s) * width) & (yy >= v * height) &
               (yy < (v + s) * height))
        disparity = torch.where(box & (disparity < d), d, disparity)
    right = texture[:, nearest:nearest + width]
    at = (x - disparity + nearest).clamp(0, width + 2 * nearest - 2)
    low = at.floor()
    part = at - low
    left = (torch.gather(texture, 1, low.long()) * (1 - part) +
            torch.gather(texture, 1, low.long() + 1) * part)

    def seen(image):
        image = image + 2.0 * torch.randn(image.shape, generator=gen, device="cuda")
        return image.round().clamp(0, 255).to(torch.uint8).contiguous()

    return seen(left), seen(right)


def _nearest(disparities):
    return min(120, disparities - 8)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _frames(case, seed):
    """The raw host frames of `pairs` pairs seen by the same rig."""
    width, height = case["width"], case["height"]
    rig, gen, pairs = scene.rig(width, height), _generator(seed), []
    for _ in range(case["pairs"]):
        left, right = _pair(width, height, gen, _nearest(case["disparities"]))
        frames = scene.raw_frames(left.cpu().numpy(), right.cpu().numpy(), rig)
        pairs.append(dict(zip(segment.FRAMES, frames)))
    return rig, pairs


def _stage_inputs(case, seed):
    """Frames, a disparity map as the matcher leaves it (unmatched pixels at -1) and the
    pair's before it, with the misses counted so far."""
    width, height, gen = case["width"], case["height"], _generator(seed)
    left, right = _pair(width, height, gen, 100)

    def disparity():
        coarse = torch.rand((1, 1, height // 60 + 2, width // 60 + 2), generator=gen,
                            device="cuda")
        smooth = torch.nn.functional.interpolate(coarse, (height, width), mode="nearest")[0, 0]
        value = 4 + 100 * smooth + 0.25 * torch.randn((height, width), generator=gen,
                                                      device="cuda")
        lost = torch.rand((height, width), generator=gen, device="cuda") < 0.15
        return torch.where(lost, -1.0, value.clamp(min=0.5)).contiguous()

    missed = torch.randint(0, 4, (height, width), generator=gen, device="cuda").float()
    return left, right, disparity(), disparity(), missed


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": dict(case)}
    if kind in ("sgm", "c2f"):
        state["left"], state["right"] = _pair(case["width"], case["height"], _generator(seed),
                                              _nearest(case.get("disparities", 128)))
        shape = (case["height"], case["width"])
        state["disparity"] = torch.empty(shape, dtype=torch.float32, device="cuda")
        if kind == "c2f":
            state["base"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    elif kind == "stages":
        _prepare_stages(state, case, seed)
    elif kind in ("pipeline", "stream"):
        rig, state["pairs"] = _frames(case, seed)
        geometry = segment.standard_geometry(case["width"], case["height"], the_rig=rig)
        matcher = (stage.Disparity, {"num_disparities": case["disparities"]})
        stages = [stage.Rectification, matcher, stage.SpeckleFilter]
        stages += [stage.Depth, stage.PointCloud] if kind == "pipeline" else \
            [stage.TemporalFilter, stage.Depth, stage.Quality]
        status, members = segment.members(stages, geometry)
        assert status == "ok", members
        status, state["segment"] = segment.CudaSegment.build(members, geometry)
        assert status == "ok", state["segment"]
    else:
        shapes, gen = _batch_shapes(case), _generator(seed)
        plan = batch.BatchPlan(segment.context(0), shapes, {"engine": 1, "streams": 8})
        state["plan"], state["views"] = plan, [plan.device_views(i) for i in range(len(shapes))]
        for (w, h, settings), (left, right, _) in zip(shapes, state["views"]):
            images = _pair(w, h, gen, _nearest(settings["disparities"]))
            left.copy_(images[0])
            right.copy_(images[1])
    return state


DECIMATION, NEAREST_M, FARTHEST_M = 4, 0.05, 20.0
TEMPORAL = (0.4, 2.0, 2.0, 255.0)  # alpha, delta, hold, max_missed: the stage's defaults


def _prepare_stages(state, case, seed):
    width, height = case["width"], case["height"]
    rig = scene.rig(width, height)
    cams = scene.cameras(rig)
    left, right, disparity, before, missed = _stage_inputs(case, seed)
    state.update(
        rig=rig, frames=(left, right), matched=disparity, previous=before, missed=missed,
        quality_previous=before.clone(),
        cameras=[native.make_camera(cams[s]["k"], cams[s]["d"], cams[s]["inverse_pr"])
                 for s in ("left", "right")])
    shape = (height, width)

    def empty(dtype, *of):
        return torch.empty(of or shape, dtype=dtype, device="cuda")

    state["out"] = {
        "left": empty(torch.uint8), "right": empty(torch.uint8),
        "disparity": empty(torch.float32), "depth_mm": empty(torch.int16),
        "depth_m": empty(torch.float32),
        "grid": empty(torch.float32, height // DECIMATION, width // DECIMATION, 3),
        "points": empty(torch.int32, 1), "quality_sums": empty(torch.float32, 5),
        "missed": state["missed"], "previous": state["previous"],
        "quality_previous": state["quality_previous"]}


# ---------------------------------------------------------------- one pass
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "sgm":
        segment.context(0).sgm_device(
            state["left"].data_ptr(), state["right"].data_ptr(), case["width"], case["height"],
            state["disparity"].data_ptr(), stream=_stream(), disparities=case["disparities"],
            paths=case["paths"], p1=case["p1"], p2=case["p2"], uniqueness=case["uniqueness"])
        return state["disparity"]
    if kind == "c2f":
        segment.context(0).sgm_coarse_to_fine_device(
            state["left"].data_ptr(), state["right"].data_ptr(), case["width"], case["height"],
            state["disparity"].data_ptr(), state["base"].data_ptr(), stream=_stream(),
            band=case["band"], paths=case["paths"], census=case["census"])
        return {"disparity": state["disparity"], "base": state["base"]}
    if kind == "stages":
        return _run_stages(state, case["width"], case["height"])
    if kind == "batch":
        state["plan"].launch(stream=_stream())
        return [views[2] for views in state["views"]]
    module, seg, sent, replies = segment.CudaSegment, state["segment"], [], []

    def reply():
        got = module.await_(sent.pop(0), seg, 60000)
        assert got[0] == "ok", got
        replies.append(got[1])

    for entries in state["pairs"]:
        if len(sent) == module.depth():
            reply()
        status, request = module.send_request(entries, seg)
        assert status == "ok", request
        sent.append(request)
    while sent:
        reply()
    return replies


def _run_stages(state, width, height):
    """Rectification of a pair; a disparity map through the speckle filter, the temporal
    filter, depth and the point cloud; the quality sums against the pair before."""
    s, out, call, rig = _stream(), state["out"], native.call, state["rig"]
    frames, focal, (cx, cy) = state["frames"], rig["focal_length_px"], rig["principal_point"]
    call("nxs_rectify_pair_device", frames[0].data_ptr(), frames[1].data_ptr(), width, height,
         ctypes.byref(state["cameras"][0]), ctypes.byref(state["cameras"][1]), width, height,
         out["left"].data_ptr(), out["right"].data_ptr(), s)
    call("nxs_despeckle_device", state["matched"].data_ptr(), width, height, 12.0, 1.0, 3,
         out["disparity"].data_ptr(), s)
    call("nxs_temporal_device", out["disparity"].data_ptr(), out["previous"].data_ptr(),
         out["missed"].data_ptr(), width * height, *TEMPORAL, s)
    call("nxs_depth_device", out["disparity"].data_ptr(), width * height, focal,
         rig["baseline_m"], out["depth_mm"].data_ptr(), out["depth_m"].data_ptr(), s)
    call("nxs_cloud_device", out["depth_m"].data_ptr(), width, height, DECIMATION, focal, cx, cy,
         NEAREST_M, FARTHEST_M, out["grid"].data_ptr(), out["points"].data_ptr(), s)
    call("nxs_quality_device", out["disparity"].data_ptr(), state["quality_previous"].data_ptr(),
         width, height, out["quality_sums"].data_ptr(), s)
    return out


# ---------------------------------------------------------------- the results in 64 bits
def exact(case, seed):
    """Pipelines and streams have no such values: rectified images are whole numbers, and a
    64-bit rectification would hand the matcher other ones wherever a sample lies at a half."""
    kind = case["kind"]
    if kind == "sgm":
        left, right = _pair(case["width"], case["height"], _generator(seed),
                            _nearest(case["disparities"]))
        return _exact_sgm(left, right, case["disparities"], case["paths"], case["p1"],
                          case["p2"], case["uniqueness"])
    if kind == "c2f":
        left, right = _pair(case["width"], case["height"], _generator(seed), _nearest(128))
        return {"disparity": _exact_c2f(left, right, case["band"], case["paths"],
                                        case["census"]), "base": None}
    if kind == "stages":
        return _exact_stages(case, seed)
    if kind == "batch":
        gen, results = _generator(seed), []
        for w, h, settings in _batch_shapes(case):
            left, right = _pair(w, h, gen, _nearest(settings["disparities"]))
            results.append(_exact_sgm(left, right, settings["disparities"], settings["paths"], 8,
                                      64, UNIQUENESS))
        return results
    return None


DIRECTIONS = [(0, 1), (0, -1), (1, 0), (-1, 0), (1, 1), (1, -1), (-1, 1), (-1, -1)]


def _padded(image, rows, columns):
    return torch.nn.functional.pad(image[None, None].float(), (columns, columns, rows, rows),
                                   mode="replicate")[0, 0].int()


def _census(image, window="sparse_9x7"):
    height, width = image.shape
    padded = _padded(image, 3, 4)
    if window == "sparse_9x7":
        offsets = [(dy, dx) for dy in range(-3, 4) for dx in range(-4, 5) if dy and dx]
    else:
        offsets = [(dy, dx) for dy in range(-2, 3) for dx in range(-4, 5) if dy or dx]

    def moved(dy, dx):
        return padded[3 + dy:3 + dy + height, 4 + dx:4 + dx + width]

    centre = moved(0, 0)
    if window == "dense_9x5_blend":
        weighted = sum((2 - abs(dy)) * (2 - abs(dx)) * moved(dy, dx)
                       for dy in (-1, 0, 1) for dx in (-1, 0, 1))
        centre = (weighted + 16 * centre + 24) // 32
    code = torch.zeros((height, width), dtype=torch.int64, device=image.device)
    for bit, (dy, dx) in enumerate(offsets):
        code |= (moved(dy, dx) + 1 < centre).long() << bit
    return code


def _count(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    return ((x * 0x0101010101010101) >> 56).to(torch.int16)


def _costs(left, right, disparities, base=None):
    """costs[d] of left's pixel against right's pixel x - base - d, codes left of the image 0."""
    height, width = left.shape
    x = torch.arange(width, device=left.device)[None, :].expand(height, width)
    costs = torch.empty((height, width, disparities), dtype=torch.int16, device=left.device)
    for d in range(disparities):
        column = x - d if base is None else x - base - d
        code = torch.where(column >= 0, torch.gather(right, 1, column.clamp(min=0)), 0)
        costs[:, :, d] = _count(left ^ code)
    return costs


def _path_sums(costs, paths, p1, p2, base=None):
    """The sum of the path costs; with `base`, a pixel's candidates start at its own
    disparity and those the pixel before lacks cost p2."""
    height, width, n = costs.shape
    totals = torch.zeros_like(costs)
    for dy, dx in DIRECTIONS[:paths]:
        along = costs if dy else costs.transpose(0, 1)
        total = totals if dy else totals.transpose(0, 1)
        bases = None if base is None else base if dy else base.t()
        steps = along.shape[0]
        order = range(steps) if (dy if dy else dx) > 0 else range(steps - 1, -1, -1)
        side = dx if dy else 0
        state, before = torch.zeros_like(along[0]), None if base is None else bases[order[0]]

        def entered(t):  # each line's state at its next pixel; a line that enters has none
            if side == 0:
                return t
            t = t.roll(side, 0)
            t[0 if side > 0 else -1] = 0
            return t

        for k, i in enumerate(order):
            if k:
                state = entered(state)
            if base is None:
                near = torch.full_like(state, 1 << 12)
                near[:, 1:] = state[:, :-1]
                near[:, :-1] = torch.minimum(near[:, :-1], state[:, 1:])
                own = state
            else:
                now = bases[i]
                if k:
                    shift = now - before.roll(side, 0)
                    if side:
                        shift[0 if side > 0 else -1] = 0
                    shift = shift.clamp(-n - 1, n + 1)
                else:
                    shift = torch.zeros_like(now)
                wide = torch.nn.functional.pad(state, (n + 2, n + 2), value=p2)
                at = torch.arange(n, device=costs.device)[None, :] + shift[:, None] + n + 2
                own = torch.gather(wide, 1, at)
                near = torch.minimum(torch.gather(wide, 1, at - 1), torch.gather(wide, 1, at + 1))
                before = now
            state = torch.minimum(own, near + p1).clamp(max=p2) + along[i]
            total[i] += state
            state = state - state.amin(1, keepdim=True)
    return totals


def _select(totals, disparities, uniqueness, base=None):
    """(disparity, keys): the winner with its uniqueness test (the product in 32 bits, as the
    test is defined) and the parabola's step."""
    height, width, n = totals.shape
    x = torch.arange(width, device=totals.device)[None, :, None]
    k = torch.arange(n, device=totals.device)[None, None, :]
    disparity, keys = [], []
    rows = max(1, (1 << 26) // (width * n))
    for y in range(0, height, rows):
        start = 0 if base is None else base[y:y + rows, :, None].clamp(min=0)
        values = totals[y:y + rows].int() + ((start + k > x).int() << 15)
        lowest = (values.long() * 65536 + k).amin(2)
        minimum, winner = lowest >> 16, lowest & 65535
        second = torch.where((k - winner[:, :, None]).abs() > 1, values, 2 ** 31 - 1).amin(2)
        lower = torch.gather(values, 2, (winner - 1).clamp(min=0)[:, :, None])[:, :, 0].double()
        upper = torch.gather(values, 2, (winner + 1).clamp(max=n - 1)[:, :, None])[:, :, 0].double()
        at = winner + (start if base is None else start[:, :, 0])
        accepted = second.float() > minimum.float() * torch.tensor(uniqueness, dtype=torch.float32,
                                                                   device=totals.device)
        accepted &= at <= x[:, :, 0]
        if base is not None:
            accepted &= base[y:y + rows] >= 0
        curve = lower + upper - 2.0 * minimum
        step = ((lower - upper) / (2.0 * curve.clamp(min=1.0))).clamp(-0.5, 0.5)
        refine = (curve > 0) & (winner > 0) & (winner < n - 1)
        refine &= (at < disparities - 1) & (at < x[:, :, 0])
        value = at.double() + torch.where(refine, step, torch.zeros_like(step))
        disparity.append(torch.where(accepted, value, torch.full_like(value, -1.0)))
        keys.append(torch.where(accepted, minimum * 65536 + at, torch.full_like(at, -1)))
    return torch.cat(disparity), torch.cat(keys)


def _check_and_median(disparity, keys):
    height, width = disparity.shape
    x = torch.arange(width, device=disparity.device)[None, :].expand(height, width)
    none = 1 << 40
    winner = keys & 65535
    candidate = torch.where(keys >= 0, (keys >> 16) * 65536 + (65535 - winner), none)
    column = torch.where(keys >= 0, x - winner, 0).clamp(min=0)
    right = torch.full_like(keys, none).scatter_reduce(1, column, candidate, "amin")
    rejected = torch.ones_like(keys, dtype=torch.bool)
    for d in (disparity.floor().long(), disparity.ceil().long()):
        at = x - d
        found = torch.gather(right, 1, at.clamp(0, width - 1))
        there = 65535 - (found & 65535)
        rejected &= (at >= 0) & (at < width) & (found != none) & ((there - d).abs() > 1)
    checked = torch.where((disparity >= 0) & ~rejected, disparity,
                          torch.full_like(disparity, -1.0))
    padded = torch.nn.functional.pad(checked[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    nine = torch.stack([padded[dy:dy + height, dx:dx + width]
                        for dy in range(3) for dx in range(3)])
    return nine.sort(0).values[4]


def _exact_sgm(left, right, disparities, paths, p1, p2, uniqueness):
    totals = _path_sums(_costs(_census(left), _census(right), disparities), paths, p1, p2)
    return _check_and_median(*_select(totals, disparities, uniqueness))


def _exact_c2f(left, right, band, paths, census, margin=4, p1=8, p2=64):
    height, width = left.shape

    def half(image):
        blocks = image.int().reshape(height // 2, 2, width // 2, 2)
        return ((blocks.sum((1, 3)) + 2) // 4).to(torch.uint8)

    coarse = _exact_sgm(half(left), half(right), 64, paths, p1, p2, UNIQUENESS)
    valid = torch.where(coarse >= 0, coarse, torch.full_like(coarse, 1e9))
    lowest = -torch.nn.functional.max_pool2d(-torch.nn.functional.pad(
        valid[None, None], (1, 1, 1, 1), value=1e9), 3, 1)[0, 0]
    base = torch.where(lowest < 1e9, ((lowest * 2).floor() - margin).clamp(0, 128 - band),
                       torch.full_like(lowest, -1.0)).long()
    base = base.repeat_interleave(2, 0).repeat_interleave(2, 1)
    start = base.clamp(min=0)
    costs = _costs(_census(left, census), _census(right, census), band, start)
    totals = _path_sums(costs, paths, p1, p2, start)
    return _check_and_median(*_select(totals, 128, UNIQUENESS, base))


def _exact_stages(case, seed):
    width, height = case["width"], case["height"]
    rig = scene.rig(width, height)
    _, _, matched, before, missed = _stage_inputs(case, seed)
    c, padded = matched.double(), torch.nn.functional.pad(matched.double(), (3, 3, 3, 3), value=-1.0)
    support = torch.zeros_like(c)
    for dy in range(7):
        for dx in range(7):
            n = padded[dy:dy + height, dx:dx + width]
            if (dy, dx) != (3, 3):  # the difference in 32 bits, as the filter's test takes it
                support += (n > 0) & ((n.float() - matched).abs() <= 1.0)
    kept = torch.where((c > 0) & (support >= 12), c, torch.full_like(c, -1.0))
    alpha, delta, hold, most = TEMPORAL
    previous, matches = before.double(), kept > 0
    agree = matches & (previous > 0) & ((kept.float() - before).abs() <= delta)
    # the weights are 32-bit settings
    weight = float(np.float32(alpha))
    rest = float(np.float32(1.0) - np.float32(alpha))
    smoothed = torch.where(agree, weight * kept + rest * previous, kept)
    misses = torch.where(matches, torch.zeros_like(kept), missed.double() + 1)
    held = ~matches & (previous > 0) & (misses <= hold)
    filtered = torch.where(held, previous, smoothed)
    focal_baseline = float(np.float32(rig["focal_length_px"])) * float(np.float32(rig["baseline_m"]))
    positive = filtered > 0
    depth = torch.where(positive, focal_baseline / torch.where(positive, filtered, 1.0), 0.0)
    z = depth[:height // DECIMATION * DECIMATION:DECIMATION,
              :width // DECIMATION * DECIMATION:DECIMATION]
    # the range's ends are 32-bit settings
    inside = (z.float() > np.float32(NEAREST_M).item()) & (z.float() < FARTHEST_M)
    v = torch.arange(z.shape[0], device="cuda", dtype=torch.float64)[:, None] * DECIMATION
    u = torch.arange(z.shape[1], device="cuda", dtype=torch.float64)[None, :] * DECIMATION
    cx, cy = rig["principal_point"]
    over = z / float(np.float32(rig["focal_length_px"]))
    grid = torch.stack([(u - cx) * over, (v - cy) * over, z], -1)
    grid = torch.where(inside[:, :, None], grid, torch.full_like(grid, float("nan")))
    seen = (filtered > 0).double()
    both = seen * (previous > 0)
    sums = torch.stack([seen.sum(), (filtered * seen).sum(), (filtered * filtered * seen).sum(),
                        both.sum(), ((filtered - previous).abs() * both).sum()])
    return {"left": None, "right": None, "disparity": filtered, "depth_mm": None,
            "depth_m": depth, "grid": grid, "points": None, "quality_sums": sums,
            "missed": misses.clamp(max=most), "previous": filtered,
            "quality_previous": filtered}
