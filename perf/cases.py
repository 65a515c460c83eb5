"""Cases for timing the framework's public entry points on a B200.

What a user runs: one scan already in device memory (``fx_process_device``),
several scans in flight (``batch.run_device_batch``), a job with host arrays
(``process_b200``), the at-floor routing census with its JSON
(``routing.route_at_floor_mask``, ``routing.serialize_routing_json``), and
the producer records alone (``fx_producer_rows_static``).  Sizes are those of
the repository's benchmark and tests: 256 x 256 crops, 512 x 512, 1024 x 768,
2892 x 1973, 5782 x 3946 and its transpose, and odd crops in between.

Scans are made on the GPU from the seed with the statistics of
``synthetic.py``: smooth colour fields with grain, IR near 52000, and discs,
scratches and dense blobs that darken both.
"""

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.getcwd(), "digital-fauxice_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from fauxice_b200 import _lib, batch, contracts, engine, routing, synthetic  # noqa: E402
from fauxice_b200.profile import DEFAULT_PROFILE, NIKON_PE_INITIAL_STATE  # noqa: E402

FULL = synthetic.FULL_FRAME
DAMAGE = {"native": synthetic.NATIVE_FRAME, "heavy": synthetic.HEAVY_FULL}


def listed():
    return [
        # the smallest scan the tests take whole: launches and short chains
        {"name": "frame_256", "kind": "frame", "h": 256, "w": 256, "coverage": 0.06,
         "damage": "native", "planes": False},
        # an odd crop of the serving range (256..2048 a side), lightly
        # damaged, with the score plane and the changed mask asked for
        {"name": "frame_odd_planes", "kind": "frame", "h": 1487, "w": 903, "coverage": 0.015,
         "damage": "native", "planes": True},
        # the half-size frame: three requests in ten of the serving workload
        {"name": "frame_half", "kind": "frame", "h": 2892, "w": 1973, "coverage": 0.06,
         "damage": "native", "planes": False},
        # the headline: one native 4000 dpi frame
        {"name": "frame_native", "kind": "frame", "h": 5782, "w": 3946, "coverage": 0.06,
         "damage": "native", "planes": False},
        # heavy damage at full size (dense blobs, crossing scratches)
        {"name": "frame_heavy", "kind": "frame", "h": 5782, "w": 3946, "coverage": 0.05,
         "damage": "heavy", "planes": False},
        # a roll of uneven scans and orientations, four in flight
        {"name": "batch_mix", "kind": "batch", "scale": 1.0, "coverage": 0.06,
         "damage": "native", "slots": 4},
        # host arrays in and out with diagnostics, small crop
        {"name": "job_512", "kind": "job", "h": 512, "w": 512, "coverage": 0.06,
         "damage": "native", "planes": True},
        # host arrays in and out, native frame: copies and the output SHA-256
        {"name": "job_native", "kind": "job", "h": 5782, "w": 3946, "coverage": 0.06,
         "damage": "native", "planes": False},
        # the routing census of a small odd crop's at-floor mask
        {"name": "census_odd", "kind": "census", "h": 701, "w": 933, "coverage": 0.06,
         "damage": "native"},
        # the routing census of a native frame's at-floor mask
        {"name": "census_native", "kind": "census", "h": 5782, "w": 3946, "coverage": 0.06,
         "damage": "native"},
        # the producer records of a native frame, for callers without a context slot
        {"name": "producer_native", "kind": "producer", "h": 5782, "w": 3946, "coverage": 0.06,
         "damage": "native"},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "batch", "job", "census", "producer"))
    damage = rng.choice(("native", "native", "heavy"))
    case = {"kind": kind, "damage": damage,
            "coverage": round(math.exp(rng.uniform(math.log(0.001), math.log(0.06))), 4)}
    if kind == "batch":
        case.update(scale=round(math.exp(rng.uniform(math.log(0.1), 0.0)), 3),
                    slots=rng.choice((2, 4)))
        return case
    # sides over the whole range, either orientation, within a full frame's pixels
    long_side = _log_uniform(rng, 96, FULL[0])
    short_side = max(64, int(long_side * rng.uniform(0.45, FULL[1] / FULL[0])))
    h, w = (long_side, short_side) if rng.random() < 0.6 else (short_side, long_side)
    case.update(h=h, w=w)
    if kind in ("frame", "job"):
        case["planes"] = rng.random() < 0.4
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _spec(case, h, w):
    """Defect counts for the frame: the named damage scaled to its area, and
    the native mix further to the case's coverage."""

    spec = synthetic.scaled_spec(DAMAGE[case["damage"]], h, w)
    factor = case["coverage"] / synthetic.NATIVE_COVERAGE if case["damage"] == "native" else 1.0
    return spec, max(1, round(spec.discs * factor)), max(1, round(spec.scratches * factor))


def _stamp(plane_ir, plane_rgb, h, w, cy, cx, radius, ir, rgb):
    """Darken discs: each pixel keeps the strongest factor that covers it."""

    dev = plane_ir.device
    reach = int(math.ceil(float(radius.max())))
    span = torch.arange(-reach, reach + 1, device=dev)
    dy, dx = torch.meshgrid(span, span, indexing="ij")
    dy, dx = dy.reshape(-1), dx.reshape(-1)
    for k in range(0, len(cy), 4096):
        y = torch.as_tensor(cy[k:k + 4096], device=dev).long()[:, None] + dy
        x = torch.as_tensor(cx[k:k + 4096], device=dev).long()[:, None] + dx
        r = torch.as_tensor(radius[k:k + 4096], device=dev).float()[:, None]
        keep = (dy * dy + dx * dx)[None, :] <= r * r
        keep &= (y >= 0) & (y < h) & (x >= 0) & (x < w)
        at = (y * w + x)[keep]
        for plane, factor in ((plane_ir, ir), (plane_rgb, rgb)):
            f = torch.as_tensor(factor[k:k + 4096], device=dev).float()[:, None].expand_as(keep)
            plane.view(-1).scatter_reduce_(0, at, f[keep], "amin")


def _defects(case, h, w, seed):
    """(IR factor, RGB factor) planes of the frame's defects."""

    rng = np.random.default_rng(seed)
    spec, discs, scratches = _spec(case, h, w)
    ir = torch.ones((h, w), device="cuda")
    rgb = torch.ones((h, w), device="cuda")
    groups = [(discs, spec.disc_radius, spec.ir_factor),
              (spec.blobs, spec.blob_radius, spec.blob_ir_factor)]
    for count, radius, factor in groups:
        if count:
            _stamp(ir, rgb, h, w, rng.uniform(0, h, count), rng.uniform(0, w, count),
                   rng.uniform(*radius, count), rng.uniform(*factor, count),
                   rng.uniform(*spec.rgb_factor, count))
    ys, xs, rs, irs, rgbs = [], [], [], [], []
    for _ in range(scratches):
        length = rng.uniform(*spec.scratch_length)
        n = int(2 * length) + 2
        heading = rng.uniform(0, 2 * np.pi) + np.cumsum(rng.normal(0.0, 0.02, n))
        ys.append(rng.uniform(0, h) + np.cumsum(0.5 * np.sin(heading)))
        xs.append(rng.uniform(0, w) + np.cumsum(0.5 * np.cos(heading)))
        rs.append(np.full(n, int(rng.integers(1, 4)) / 2.0))
        irs.append(np.full(n, rng.uniform(*spec.ir_factor)))
        rgbs.append(np.full(n, rng.uniform(*spec.rgb_factor)))
    _stamp(ir, rgb, h, w, np.floor(np.concatenate(ys)), np.floor(np.concatenate(xs)),
           np.concatenate(rs), np.concatenate(irs), np.concatenate(rgbs))
    return ir, rgb


def _scan(case, h, w, seed):
    """One H x W x 4 RGBI scan on the device, 16-bit samples in an int16 tensor."""

    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed + 1)
    ir, rgb = _defects(case, h, w, seed + 2)
    y = (torch.arange(h, device="cuda", dtype=torch.float32) / h)[:, None]
    x = (torch.arange(w, device="cuda", dtype=torch.float32) / w)[None, :]
    out = torch.empty((h, w, 4), dtype=torch.int16, device="cuda")
    for c in range(4):
        if c < 3:
            plane = torch.full((h, w), 30000.0, device="cuda")
            for a in rng.dirichlet((2.0, 2.0, 2.0)) * 12000.0:
                fy, fx = rng.uniform(0.5, 3.0, 2) * rng.choice((-1.0, 1.0), 2)
                plane += a * torch.sin(2 * math.pi * (fy * y + fx * x)
                                       + rng.uniform(0, 2 * math.pi))
        else:
            plane = torch.full((h, w), 52000.0, device="cuda")
        plane += torch.randn((h, w), generator=gen, device="cuda") * (600.0 if c < 3 else 400.0)
        plane *= rgb if c < 3 else ir
        out[..., c] = plane.clamp_(0.0, 65535.0).round_().to(torch.int32).to(torch.int16)
    return out


def _mask(case, h, w, seed):
    """An at-floor mask: the pixels of the deep defects, as the score plane's
    floor marks them."""

    ir, _ = _defects(case, h, w, seed)
    return ir < 0.6


def _batch_shapes(case):
    return [(max(8, round(h * case["scale"])), max(8, round(w * case["scale"])))
            for h, w in synthetic.BATCH_SHAPES]


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "ctx": engine.context(0),
             "params": DEFAULT_PROFILE.hot_path_parameters().to_c()}
    if kind == "batch":
        state["slots"] = case["slots"]
        state["scans"] = [_scan(case, h, w, 1000 * seed + k)
                          for k, (h, w) in enumerate(_batch_shapes(case))]
        state["outs"] = [torch.empty((*s.shape[:2], 3), dtype=torch.int16, device="cuda")
                         for s in state["scans"]]
        state["frames"] = [batch.DeviceFrame(s.data_ptr(), s.shape[0], s.shape[1], o.data_ptr())
                           for s, o in zip(state["scans"], state["outs"])]
    elif kind == "census":
        state["mask"] = _mask(case, case["h"], case["w"], 1000 * seed)
    elif kind == "job":
        main = _scan(case, case["h"], case["w"], 1000 * seed).cpu().numpy().view(np.uint16)
        frame = contracts.RGBI16Frame
        state["job"] = contracts.ProcessingJob(
            acquisition=contracts.DualRGBIAcquisition(
                prepass=frame(synthetic.make_prepass(main), contracts.AcquisitionEpoch.PREPASS,
                              285, "prepass"),
                main=frame(main, contracts.AcquisitionEpoch.MAIN, 4000, "main"),
                same_frame_id="scan"),
            scanner_model=contracts.ScannerModel.NIKON_SUPER_COOLSCAN_5000_ED,
            mode=contracts.ProcessingMode.NORMAL, selector=8, resolution_metric=4000,
            bit_depth=16, focus_exposure_locked=True)
        state["planes"] = case["planes"]
    else:
        h, w = case["h"], case["w"]
        state["scan"] = _scan(case, h, w, 1000 * seed)
        if kind == "frame":
            state["out"] = torch.empty((h, w, 3), dtype=torch.int16, device="cuda")
            if case["planes"]:
                state["score"] = torch.empty((h, w), dtype=torch.float32, device="cuda")
                state["changed"] = torch.empty((h, w), dtype=torch.uint8, device="cuda")
        else:
            state["rows"] = torch.empty((4, h), dtype=torch.float32, device="cuda")
            state["stages"] = torch.empty((h + 6, 8), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the library works on its own streams
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------


def _counts(c):
    return [c.attempted, c.written, c.public_advances, c.changed, c.final_state,
            c.startup_final_state, *c.startup_attempted, *c.startup_advances, c.rng_dependent]


def _pointer(tensor):
    return None if tensor is None else ctypes.c_void_p(tensor.data_ptr())


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "frame":
        scan, score, changed = state["scan"], state.get("score"), state.get("changed")
        counters = _lib.FxCounters()
        ctx.check(_lib.load().fx_process_device(
            ctx.handle, _pointer(scan), scan.shape[0], scan.shape[1],
            ctypes.byref(state["params"]), None, NIKON_PE_INITIAL_STATE, _pointer(state["out"]),
            _pointer(score), _pointer(changed), None, ctypes.byref(counters)))
        return {"rgb": state["out"], "counts": np.array(_counts(counters), np.int64),
                "score": score, "changed": changed}
    if kind == "batch":
        counters = batch.run_device_batch(ctx, state["frames"], slots=state["slots"],
                                          params=state["params"])
        return {"rgb": state["outs"],
                "counts": np.array([_counts(c) for c in counters], np.int64)}
    if kind == "job":
        result = engine.process_b200(state["job"], export_diagnostics=state["planes"])
        r = result.replay
        out = {"rgb": result.output_rgb16.view(np.int16),
               "counts": np.array([r.attempted_pixels, r.written_pixels, r.public_rng_advances,
                                   r.changed_pixels, r.final_rng_state], np.int64),
               "sha256": np.frombuffer(bytes.fromhex(r.output_sha256), np.uint8)}
        if state["planes"]:
            d = result.diagnostics
            out.update(score=d.score_plane, at_floor=d.at_floor_mask, changed=d.changed_mask)
        return out
    if kind == "census":
        result = routing.route_at_floor_mask(state["mask"])
        text = routing.serialize_routing_json(result)
        # the document in a buffer whose size depends on the frame alone
        document = np.zeros(65536 + result.synthesis_mask.size // 8, np.uint8)
        document[:len(text)] = np.frombuffer(text, np.uint8)
        return {"provisional": result.provisional_labels, "synthesis": result.synthesis_mask,
                "final": result.final_labels, "json": document, "json_bytes": len(text)}
    scan = state["scan"]
    ctx.check(_lib.load().fx_producer_rows_static(
        ctx.handle, _pointer(scan), scan.shape[0], scan.shape[1], _pointer(state["rows"]),
        _pointer(state["stages"]), None))
    return {"rows": state["rows"], "stages": state["stages"]}


def work(case):
    """Bytes in and out once; operations of the per-pixel chains on the half
    of the pixels that are attempted (five 9x9 averages at three scales, the
    combiner, up to two draws a channel)."""

    if case["kind"] == "batch":
        px = sum(h * w for h, w in _batch_shapes(case))
        return {"bytes": 14.0 * px, "flops": 180.0 * px}
    px = case["h"] * case["w"]
    if case["kind"] == "census":
        return {"bytes": 10.0 * px, "flops": 0.0}
    if case["kind"] == "producer":
        return {"bytes": 8.0 * px, "flops": 10.0 * px}
    planes = 0 if not case["planes"] else (5 if case["kind"] == "frame" else 6)
    return {"bytes": (14.0 + planes) * px, "flops": 180.0 * px}


# ---------------------------------------------------------------------------
# The float outputs in 64 bits
# ---------------------------------------------------------------------------


def _quadrants(cells):
    """4x4 quadrant means of ... x 8 x 8 cells, less their mean."""

    q = cells.reshape(*cells.shape[:2], 2, 4, 2, 4).mean((3, 5)).reshape(*cells.shape[:2], 4)
    return q - q.mean(-1, keepdim=True)


def _records(scan):
    """Per-row (p1, p2, mean visible, mean infrared) of a scan: the weighted
    cumulative means of the samples before each cell's first dark IR sample,
    and the scale epochs of the whole cells."""

    raw = (scan.to(torch.int32) & 0xFFFF).double()
    h, w = raw.shape[:2]
    aw, ph = w // 8 * 8, (h + 7) // 8 * 8
    vis, ir = raw[:, :aw, 0], raw[:, :aw, 3]
    log = lambda v: 65535.0 * torch.log2(v + 1.0) / 16.0  # noqa: E731

    def cells(v, fill):  # rows padded to whole cells: blocks x cells x 8 x 8
        v = torch.nn.functional.pad(v, (0, 0, 0, ph - h), value=fill)
        return v.reshape(ph // 8, 8, aw // 8, 8).transpose(1, 2)

    passing = cells(ir, 65535.0) > 8847.2255859375
    before = passing.flatten(2).long().cumprod(-1).reshape(passing.shape).bool()
    before = before.transpose(1, 2).reshape(ph, aw)[:h]
    weight = torch.where(before, ir * ir, 0.0)
    total = weight.sum(1).cumsum(0)
    mean = [(weight * log(v)).sum(1).cumsum(0) / total for v in (vis, ir)]
    mean = [torch.where(total > 0, m, start)
            for m, start in zip(mean, (46618.78515625, 56239.65625))]
    whole = passing.flatten(2).all(-1, keepdim=True)
    dv, di = _quadrants(cells(log(vis), 0.0)), _quadrants(cells(log(ir), 0.0))
    ratio = torch.where(dv != 0, di / dv, 0.0)
    gain = torch.where((ratio < -0.125) | (ratio > 0.425), 0.0,
                       torch.where((ratio < 0) | (ratio > 0.3), 0.5 ** 0.5, 1.0))
    term = torch.where(whole, (dv * gain * cells(ir, 0.0).sum((-1, -2))[..., None]) ** 2, 0.0)
    den, num = (t.sum((1, 2))[:h // 8].cumsum(0) for t in (term, ratio * term))
    scale = torch.full((h,), 0.15, dtype=torch.float64, device=scan.device)
    first = torch.full((h,), 0.15, dtype=torch.float64, device=scan.device)
    epoch = (torch.arange(h, device=scan.device) + 1) // 8 - 1
    done = (epoch >= 0) & (den.numel() > 0)
    if den.numel():
        got = torch.where(den != 0, num / den, 0.15)[epoch.clamp(min=0)]
        defined = done & (den[epoch.clamp(min=0)] != 0)
        scale = torch.where(defined, got, scale)
        first = torch.where(defined, 1.5 * got, first)
    return torch.stack([first, scale, mean[0], mean[1]])


def _score(scan):
    """The score plane: the stage's infrared residual of each pixel, the
    smallest of three neighbours, scaled and clipped."""

    raw = (scan.to(torch.int32) & 0xFFFF).double()
    h, w = raw.shape[:2]
    _, p2, mv, mi = _records(scan)
    row = torch.arange(h, device=scan.device)
    alpha, nxt = p2[row][:, None], (row + 1).clamp(max=h - 1)
    base = ((mi - mv * p2) / (1.0 - p2))[nxt][:, None]
    vis, ir = (65535.0 * torch.log2(raw[..., c] + 1.0) / 16.0 for c in (0, 3))
    aux = (ir - alpha * vis) / (1.0 - alpha) - 1.0
    sample = aux.clone()
    sample[:, 1:-1] = torch.minimum(torch.minimum(aux[:, :-2], aux[:, 1:-1]), aux[:, 2:])
    p = DEFAULT_PROFILE.hot_path_parameters()
    score = ((base + p.score_addend) - sample) * p.score_scale + p.score_offset
    return score.clamp(p.score_floor, 1.0)


def exact(case, seed):
    """Float outputs only: the rest are whole numbers and bytes."""

    kind = case["kind"]
    if kind == "producer":
        scan = _scan(case, case["h"], case["w"], 1000 * seed)
        return {"rows": _records(scan), "stages": None}
    if kind in ("frame", "job") and case["planes"]:
        score = _score(_scan(case, case["h"], case["w"], 1000 * seed))
        if kind == "frame":
            return {"rgb": None, "counts": None, "score": score, "changed": None}
        return {"rgb": None, "counts": None, "sha256": None, "score": score.cpu().numpy(),
                "at_floor": None, "changed": None}
    return None
