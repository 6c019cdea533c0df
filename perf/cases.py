"""The renderer's work as a user's program has it done, for timing and comparing builds.

A case is a dict of plain values; `op` names the call:

  viewer    Application.step(): the headless viewer's frame (the Cornell box)
  pt        rr_pathtracer_execute + rr_accumulate_execute: reference frames
  di        rr_restir_di_execute with history
  gi, rpt   ReSTIRGIPass / ReSTIRPTPass.execute over ReSTIR DI's G-buffer
  atrous    rr_atrous_execute
  guided    a guided frame: rr_guided_pathtracer_execute, accumulate, rr_guide_update
  train     one training step of the learned guide on another integrator's samples
  eval      the learned guide evaluated at surface points
  batch     rr_batch_execute: many small scenes in one set of (captured) launches

A renderer keeps its context and its scenes over many frames and cameras, so
these are made once per process (`_context`, `_scene`); the images, passes,
guides, cameras and frame seeds are made anew by prepare().
"""
import ctypes as C
import functools
import math
import weakref

import numpy as np
import torch

from research_b200 import passes, rr

ROOM_SEED = 0x5EED0002          # the benchmark's room
BOUNDS = 20.5                   # guide bounds around the room (box half-size 20)
VIEW_HEIGHT = 1080


def listed():
    return [
        # the smallest frame: an interactive preview of the default scene, one
        # path per pixel, accumulating (launches and host work count)
        {"name": "viewer_preview", "op": "viewer", "width": 256, "height": 256, "mode": "pt"},
        # the viewer at its default window size with its realtime passes:
        # ReSTIR DI + GI, denoised
        {"name": "viewer_realtime", "op": "viewer", "width": 1280, "height": 720, "mode": "di+gi+denoise"},
        # the benchmark's reference frame: 1M triangles, 1080p, 4 paths per pixel
        {"name": "pt_1080p", "op": "pt", "width": 1920, "height": 1080, "triangles": 1_000_000, "spp": 4,
         "bounces": 5, "emitters": 0},
        # a smaller scene lit by its emissive triangles alone, emitter sampling
        # on, an odd window size
        {"name": "pt_emitters_odd", "op": "pt", "width": 641, "height": 359, "triangles": 100_000, "spp": 2,
         "bounces": 5, "emitters": 1},
        # the benchmark's ReSTIR DI frame: 32 candidates, 5 neighbours in 30 pixels
        {"name": "di_1080p", "op": "di", "width": 1920, "height": 1080, "triangles": 1_000_000, "candidates": 32,
         "neighbors": 5, "radius": 30, "emitters": 0},
        # indirect light with the reuse passes' default settings
        {"name": "gi_720p", "op": "gi", "width": 1280, "height": 720, "triangles": 1_000_000},
        {"name": "rpt_1080p", "op": "rpt", "width": 1920, "height": 1080, "triangles": 1_000_000},
        # the denoiser alone, default settings
        {"name": "atrous_1080p", "op": "atrous", "width": 1920, "height": 1080, "iterations": 5, "tma": 1},
        # guided rendering of the 64 x 64 centre crop, 256 paths per pixel a
        # frame, the guide trained after each frame: both guides
        {"name": "guided_grid", "op": "guided", "guide": "grid", "side": 64, "spp": 256, "triangles": 1_000_000},
        {"name": "guided_mlp", "op": "guided", "guide": "mlp", "side": 64, "spp": 256, "triangles": 1_000_000},
        # a full batch of the learned guide's training on given samples
        {"name": "train_256k", "op": "train", "samples": 1 << 18},
        # many small scenes at once: launch-bound without batching
        {"name": "batch_32_small", "op": "batch", "scenes": 32, "side": 128, "spp": 1, "bounces": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, most):
    """An image of any size (odd ones too) between 64 x 64 and `most` pixels, 1:1 to 2:1."""
    pixels = math.exp(rng.uniform(math.log(64 * 64), math.log(most)))
    w = int(math.sqrt(pixels * rng.uniform(1.0, 2.0)))
    return {"width": w, "height": max(32, int(pixels / w))}


def draw(rng):
    op = rng.choice(["viewer", "pt", "pt", "di", "gi", "rpt", "atrous", "guided", "train", "eval", "batch"])
    tris = _log_int(rng, 10_000, 1_000_000)
    if op == "viewer":
        return {"op": op, **_size(rng, 1280 * 720), "mode": rng.choice(["pt", "di", "di+denoise", "di+gi+denoise"])}
    if op == "pt":
        return {"op": op, **_size(rng, 1920 * 1080), "triangles": tris, "spp": rng.randint(1, 4),
                "bounces": rng.randint(1, 6), "emitters": rng.randint(0, 1)}
    if op == "di":
        return {"op": op, **_size(rng, 1920 * 1080), "triangles": tris, "candidates": rng.choice([8, 16, 32]),
                "neighbors": rng.randint(1, 5), "radius": rng.randint(4, 30), "emitters": rng.randint(0, 1)}
    if op == "gi":
        return {"op": op, **_size(rng, 1280 * 720), "triangles": tris}
    if op == "rpt":
        return {"op": op, **_size(rng, 1280 * 720), "triangles": tris}
    if op == "atrous":
        return {"op": op, **_size(rng, 1920 * 1080), "iterations": rng.randint(1, 7), "tma": rng.randint(0, 1)}
    if op == "guided":
        return {"op": op, "guide": rng.choice(["grid", "mlp"]), "side": rng.randint(32, 128),
                "spp": _log_int(rng, 4, 64), "triangles": tris}
    if op == "train":
        return {"op": op, "samples": _log_int(rng, 200, 1 << 18)}
    if op == "eval":
        return {"op": op, "points": _log_int(rng, 100, 1 << 20)}
    return {"op": op, "scenes": rng.randint(2, 32), "side": rng.randint(32, 256), "spp": rng.randint(1, 2),
            "bounces": rng.randint(2, 5)}


# ── what a program keeps ───────────────────────────────────────────────────
@functools.lru_cache(maxsize=None)
def _context(tma=1):
    ctx = rr.Context(0)
    ctx.check(rr.lib().rr_atrous_set_tma(ctx.handle, tma))
    return ctx


@functools.lru_cache(maxsize=None)
def _scene(triangles, emitters=0, seed=ROOM_SEED):
    host = rr.HostScene.procedural(seed=seed, target_triangles=triangles,
                                   emissive_triangles=max(16, triangles * 4096 // 1_000_000),
                                   flags=rr.SCENE_NO_EMITTER_LIGHTS if emitters else 0)
    scene = rr.Scene(_context(), host.arrays)
    host.close()
    return scene


class State:
    pass


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _images(h, w, n=None):
    return torch.zeros((h, w, 4) if n is None else (n, h, w, 4), device="cuda")


def _desc(case, angle, width=None, height=None):
    w, h = width or case["width"], height or case["height"]
    return rr.camera_desc(w, h, eye=(34.0 * math.sin(angle), 4.0, 34.0 * math.cos(angle)), center=(0.0, -3.0, 0.0))


def _guide(kind, batch, max_samples, seed):
    d = rr.GuideDesc(rr.GUIDE_GRID if kind == "grid" else rr.GUIDE_MLP, 64, 0.5, 0.9,
                     (C.c_float * 3)(*([-BOUNDS] * 3)), (C.c_float * 3)(*([BOUNDS] * 3)), max_samples, batch, 1e-2,
                     seed & 0x7FFFFFFF)
    h = C.c_void_p()
    ctx = _context()
    ctx.check(rr.lib().rr_guide_create(ctx.handle, C.byref(d), C.byref(h)))
    return h


def _layers():
    return [(80, 64), (64, 64), (64, 64), (64, 64), (64, 48)]


def _mlp_inputs(n, seed):
    """Network weights, and n path vertices with a sampled direction and its weight each."""
    g = np.random.default_rng(seed)
    params = []
    for i, o in _layers():
        params += [g.normal(size=o * i) * math.sqrt(2.0 / i), g.normal(size=o) * 0.05]
    params = np.concatenate(params).astype(np.float32)

    def unit(v):
        return v / np.linalg.norm(v, axis=1, keepdims=True)

    s = np.zeros((n, 16), np.float32)
    s[:, 0:3] = g.uniform(-BOUNDS, BOUNDS, (n, 3))
    s[:, 3] = g.lognormal(0.0, 1.0, n)
    s[:, 8:11] = unit(g.normal(size=(n, 3)))
    s[:, 4:7] = unit(s[:, 8:11] + 0.6 * g.normal(size=(n, 3)))       # around the normal
    s[:, 7] = np.arange(n, dtype=np.uint32).view(np.float32)
    s[:, 12:15] = unit(s[:, 8:11] + 0.8 * g.normal(size=(n, 3)))
    return params, s


def _noisy_frame(w, h, seed):
    """A denoiser's input: a closed room with three balls seen from inside
    (position and distance, unit normal) under noisy direct light, and a
    window to the sky (G-buffer misses)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    y, x = torch.meshgrid((torch.arange(h, device="cuda") + 0.5) / h - 0.5,
                          (torch.arange(w, device="cuda") + 0.5) / w - 0.5, indexing="ij")
    d = torch.stack([x * 1.6 * w / h, -1.6 * y, -torch.ones_like(x)], -1)
    d = d / d.norm(dim=-1, keepdim=True)
    half = torch.tensor([10.0, 6.0, 14.0], device="cuda")
    tp = half * torch.where(d < 0, -1.0, 1.0) / torch.where(d.abs() < 1e-6, 1e-6 * torch.ones_like(d), d)
    t, axis = tp.abs().min(-1)
    n = -torch.nn.functional.one_hot(axis, 3).float() * torch.sign(d)
    for c, r in (((-4.0, -3.0, -9.0), 2.5), ((3.0, -4.0, -7.0), 2.0), ((1.0, 1.0, -11.0), 1.5)):
        c = torch.tensor(c, device="cuda")
        b = (d * c).sum(-1)
        disc = b * b - (c * c).sum() + r * r
        ts = b - disc.clamp(min=0).sqrt()
        hit = (disc > 0) & (ts > 0) & (ts < t)
        t = torch.where(hit, ts, t)
        n = torch.where(hit[..., None], (d * t[..., None] - c) / r, n)
    p = d * t[..., None]
    to = torch.tensor([0.0, 5.5, -6.0], device="cuda") - p
    light = 40.0 * ((n * to).sum(-1) / to.norm(dim=-1) ** 3).clamp(min=0)
    noise = -torch.rand((h, w, 3), device="cuda", generator=g).clamp(min=1e-6).log()
    rad = light[..., None] * noise * torch.tensor([0.8, 0.7, 0.6], device="cuda")
    sky = (p[..., 2] < -13.99) & (p[..., 0].abs() < 3.0) & (p[..., 1].abs() < 2.0)
    one = torch.ones((h, w, 1), device="cuda")
    pos = torch.cat([p, t[..., None]], -1)
    pos = torch.where(sky[..., None], torch.tensor([0.0, 0.0, 0.0, -1.0], device="cuda"), pos)
    nrm = torch.cat([torch.where(sky[..., None], torch.zeros_like(n), n), one], -1)
    return torch.cat([rad, one], -1).contiguous(), pos.contiguous(), nrm.contiguous()


# ── prepare ────────────────────────────────────────────────────────────────
def prepare(case, seed):
    s = State()
    s.case, s.op = case, case["op"]
    s.frame_seed = (seed * 7919) & 0x3FFFFFFF
    s.frame = 0
    angle = 0.4 * math.sin(seed * 1.618 + 0.5)
    if s.op == "viewer":
        app = passes.Application()
        app.initialize(case["width"], case["height"])
        app.set_camera_look_at((0.6 * math.sin(seed), 1.0 + 0.2 * math.cos(seed), 3.2), (0.0, 1.0, 0.0))
        for name in case["mode"].split("+"):
            if name != "pt":
                app.set_pass_enabled({"di": "restir_di", "gi": "restir_gi"}.get(name, name), True)
        app.pathtracer.frame_count = s.frame_seed & 0xFFFF
        s.app = app
        s.end = weakref.finalize(s, app.shutdown)
    elif s.op == "pt":
        s.scene = _scene(case["triangles"], case["emitters"])
        s.cam = rr.camera_data(_desc(case, angle))
        s.radiance = _images(case["height"], case["width"], case["spp"])
        s.accumulated = _images(case["height"], case["width"])
    elif s.op in ("di", "gi", "rpt"):
        s.scene = _scene(case["triangles"], case.get("emitters", 0))
        # a slowly turning camera: the history is reprojected
        s.descs = [_desc(case, angle + 0.002 * k) for k in range(2)]
        h, w = case["height"], case["width"]
        s.pos, s.nrm, s.direct = _images(h, w), _images(h, w), _images(h, w)
        s.res = [_images(h, w), _images(h, w)]
        s.indirect = None
        if s.op != "di":
            s.indirect = (passes.ReSTIRGIPass if s.op == "gi" else passes.ReSTIRPTPass)(_context(), (w, h))
            s.indirect.frame_count = s.frame_seed & 0xFFFF
        _reuse_frame(s, rr.camera_data(s.descs[0]), True)   # the frame before
        s.cam = rr.camera_data(s.descs[1], s.descs[0])
        if s.indirect is not None:
            _direct(s, s.cam)
    elif s.op == "atrous":
        s.input, s.pos, s.nrm = _noisy_frame(case["width"], case["height"], seed)
        s.ping = [_images(case["height"], case["width"]) for _ in range(2)]
    elif s.op == "guided":
        side = case["side"]
        s.scene = _scene(case["triangles"])
        d = _desc(case, angle, side, side)
        # the crop's own camera: the full view's field of view narrowed to it
        d.fov_y_deg = 2.0 * math.degrees(math.atan(math.tan(math.radians(d.fov_y_deg) / 2.0) * side / VIEW_HEIGHT))
        s.cam = rr.camera_data(d)
        s.radiance = _images(side, side, case["spp"])
        s.accumulated = _images(side, side)
        s.params = np.zeros(rr.MLP_PARAM_COUNT, np.float32)
        s.guide = _guide(case["guide"], 1 << 18, 1 << 22, seed)
        s.end = weakref.finalize(s, rr.lib().rr_guide_destroy, s.guide)
        for _ in range(2):
            _guided_frame(s)                                # a guide that has learned something
    elif s.op == "train":
        params, samples = _mlp_inputs(case["samples"], seed)
        s.samples = torch.from_numpy(samples).cuda()
        s.params, s.grad = np.zeros_like(params), np.zeros_like(params)
        s.guide = _guide("mlp", case["samples"], case["samples"], seed)
        s.end = weakref.finalize(s, rr.lib().rr_guide_destroy, s.guide)
        _context().check(rr.lib().rr_guide_mlp_params(_context().handle, s.guide, None, None, params.ctypes.data,
                                                      rr.MLP_PARAM_COUNT, None))
    elif s.op == "eval":
        params, samples = _mlp_inputs(case["points"], seed)
        surf = np.zeros((case["points"], 3, 4), np.float32)
        surf[:, 0, :3], surf[:, 0, 3] = samples[:, 0:3], 1.0
        surf[:, 1, :3], surf[:, 1, 3] = samples[:, 8:11], 1.0
        surf[:, 2, :3] = samples[:, 12:15]
        s.surf = torch.from_numpy(surf).cuda()
        s.mix = torch.zeros((case["points"], 10, 4), device="cuda")
        s.guide = _guide("mlp", 1 << 10, 1 << 10, seed)
        s.end = weakref.finalize(s, rr.lib().rr_guide_destroy, s.guide)
        _context().check(rr.lib().rr_guide_mlp_params(_context().handle, s.guide, None, None, params.ctypes.data,
                                                      rr.MLP_PARAM_COUNT, None))
    else:
        n, side = case["scenes"], case["side"]
        # rooms of 10k to 100k triangles, evenly spread over the logarithm
        scenes = [_scene(int(10_000 * 10.0 ** (i / 32.0)), 0, ROOM_SEED + 1 + i) for i in range(n)]
        s.batch = rr.Batch(_context(), scenes)
        s.cams = [rr.camera_data(_desc(case, 0.4 * math.sin(seed + 2.4 * i), side, side)) for i in range(n)]
        s.radiance = _images(side, side, n * case["spp"]).view(n, case["spp"], side, side, 4)
        s.ptrs = [s.radiance[i].data_ptr() for i in range(n)]
    return s


# ── run ────────────────────────────────────────────────────────────────────
def _direct(s, cam):
    c = s.case
    p = rr.DIParams(s.frame_seed + s.frame, c.get("candidates", 16), 1, 1, c.get("neighbors", 4), c.get("radius", 15),
                    20, rr.DI_FLAG_EMITTERS if c.get("emitters") else 0)
    cur, prev = s.res[s.frame & 1], s.res[1 - (s.frame & 1)]
    ctx = _context()
    ctx.check(rr.lib().rr_restir_di_execute(ctx.handle, s.scene.handle, C.byref(cam), C.byref(p), s.pos.data_ptr(),
                                            s.nrm.data_ptr(), cur.data_ptr(), prev.data_ptr(), s.direct.data_ptr(),
                                            _stream()))
    s.frame += 1
    return cur


def _reuse_frame(s, cam, direct):
    if direct:
        cur = _direct(s, cam)
    if s.indirect is None:
        return {"output": s.direct, "position": s.pos, "normal": s.nrm, "reservoir": cur}
    s.indirect.execute(s.scene, cam, s.pos, s.nrm, s.direct)
    done = 1 - s.indirect.reservoir_flip
    out = {"output": s.indirect.output, "reservoir": s.indirect.reservoirs[done],
           "history": s.indirect.history[done]}
    if s.op == "rpt":
        out["guiding"] = s.indirect.guiding_fitted
    return out


def _accumulate(s, h, w, count):
    a = rr.AccParams(w, h, 0, s.frame * count)
    ctx = _context()
    ctx.check(rr.lib().rr_accumulate_execute(ctx.handle, s.radiance.data_ptr(), count, s.accumulated.data_ptr(), None,
                                             C.byref(a), _stream()))


def _guided_frame(s):
    c, ctx, L = s.case, _context(), rr.lib()
    p = rr.PtParams(s.frame_seed + s.frame * c["spp"], 5, c["spp"], 0)
    ctx.check(L.rr_guided_pathtracer_execute(ctx.handle, s.scene.handle, C.byref(s.cam), C.byref(p), s.guide,
                                             s.radiance.data_ptr(), _stream()))
    _accumulate(s, c["side"], c["side"], c["spp"])
    ctx.check(L.rr_guide_update(ctx.handle, s.guide, _stream()))
    s.frame += 1


def run(state):
    s, c, ctx, L = state, state.case, _context(), rr.lib()
    if s.op == "viewer":
        s.app.step()
        return s.app.displayed_image()
    if s.op == "pt":
        p = rr.PtParams(s.frame_seed + s.frame * c["spp"], c["bounces"], c["spp"],
                        rr.PT_FLAG_EMITTERS if c["emitters"] else 0)
        ctx.check(L.rr_pathtracer_execute(ctx.handle, s.scene.handle, C.byref(s.cam), C.byref(p),
                                          s.radiance.data_ptr(), _stream()))
        _accumulate(s, c["height"], c["width"], c["spp"])
        s.frame += 1
        return {"radiance": s.radiance, "accumulated": s.accumulated}
    if s.op in ("di", "gi", "rpt"):
        return _reuse_frame(s, s.cam, s.op == "di")
    if s.op == "atrous":
        actx = _context(c["tma"])
        p = rr.AtrousParams(c["width"], c["height"], c["iterations"], 0, 0.25, 0.20, 1.00, 0)
        slot = C.c_uint32()
        actx.check(L.rr_atrous_execute(actx.handle, s.input.data_ptr(), s.pos.data_ptr(), s.nrm.data_ptr(),
                                       s.ping[0].data_ptr(), s.ping[1].data_ptr(), C.byref(p), C.byref(slot),
                                       _stream()))
        return s.ping[slot.value]
    if s.op == "guided":
        _guided_frame(s)
        out = {"radiance": s.radiance, "accumulated": s.accumulated}
        if c["guide"] == "mlp":     # the trained weights, as a checkpoint saves them
            ctx.check(L.rr_guide_mlp_params(ctx.handle, s.guide, s.params.ctypes.data, None, None,
                                            rr.MLP_PARAM_COUNT, None))
            out["params"] = s.params
        return out
    if s.op == "train":
        ctx.check(L.rr_guide_set_samples(ctx.handle, s.guide, s.samples.data_ptr(), c["samples"], _stream()))
        ctx.check(L.rr_guide_update(ctx.handle, s.guide, _stream()))
        ctx.check(L.rr_guide_mlp_params(ctx.handle, s.guide, s.params.ctypes.data, s.grad.ctypes.data, None,
                                        rr.MLP_PARAM_COUNT, None))
        return {"params": s.params, "grad": s.grad}
    if s.op == "eval":
        ctx.check(L.rr_guide_eval(ctx.handle, s.guide, s.surf.data_ptr(), c["points"], s.mix.data_ptr(), _stream()))
        return s.mix
    s.batch.execute(s.cams, rr.PtParams(s.frame_seed + s.frame * c["spp"], c["bounces"], c["spp"], rr.PT_FLAG_GRAPH),
                    s.ptrs, _stream())
    s.frame += 1
    return s.radiance


# ── work ───────────────────────────────────────────────────────────────────
def _ray_flops(triangles):
    """A ray: one node of two boxes (40 operations) per level of a balanced tree over
    the triangles, and one triangle test."""
    return 40.0 * math.log2(2.0 * max(triangles, 2)) + 60.0


def _scene_bytes(triangles):
    """The tree and the triangles it holds, read once."""
    return triangles * (36.0 + 32.0)


def work(case):
    op = case["op"]
    n = case["width"] * case["height"] if "width" in case else 0
    t = case.get("triangles", 36)
    ray = _ray_flops(t)
    if op == "viewer":
        rays = {"pt": 10, "di": 2, "di+denoise": 2, "di+gi+denoise": 18}[case["mode"]]
        return {"bytes": 64.0 * n, "flops": n * rays * ray}
    if op == "pt":
        paths = n * case["spp"]
        return {"bytes": 16.0 * paths + 32.0 * n + _scene_bytes(t), "flops": paths * 2 * case["bounces"] * ray}
    if op == "di":      # G-buffer, reservoir, output; history read; 30 operations a candidate or neighbour
        return {"bytes": 80.0 * n + _scene_bytes(t),
                "flops": n * (2 * ray + 30.0 * (case["candidates"] + case["neighbors"]))}
    if op == "gi":
        return {"bytes": 272.0 * n + _scene_bytes(t), "flops": n * (8 * 2 + 2) * ray}
    if op == "rpt":
        return {"bytes": 304.0 * n + 3 * 16.0 * (1 << 20) + _scene_bytes(t), "flops": n * (8 * 4 * 2 + 2) * ray}
    if op == "atrous":  # 24 neighbour weights are 12 pairs: 50 operations each; 25 sums of 8
        return {"bytes": 64.0 * n, "flops": case["iterations"] * n * (12 * 50.0 + 25 * 8.0)}
    mlp = 2.0 * sum(i * o for i, o in _layers())
    if op == "guided":
        paths = case["side"] ** 2 * case["spp"]
        flops = paths * 10 * ray
        if case["guide"] == "mlp":
            flops += paths * 4 * mlp + 3.0 * (1 << 18) * mlp
        return {"bytes": 16.0 * paths + 64.0 * paths + _scene_bytes(t), "flops": flops}
    if op == "train":
        return {"bytes": 64.0 * case["samples"], "flops": 3.0 * mlp * case["samples"]}
    if op == "eval":
        return {"bytes": 208.0 * case["points"], "flops": mlp * case["points"]}
    paths = case["side"] ** 2 * case["spp"] * case["scenes"]
    return {"bytes": 16.0 * paths, "flops": paths * 2 * case["bounces"] * _ray_flops(30_000)}


# ── values in 64 bits, where the outputs have them without a renderer ──────
def _exact_atrous(case, seed):
    rad, pos, nrm = (x.double() for x in _noisy_frame(case["width"], case["height"], seed))
    h, w = case["height"], case["width"]
    sp2, sn2, sl2 = 0.25 ** 2, 0.20 ** 2, 1.0
    miss = pos[..., 3] < 0
    p = pos[..., :3]
    n = nrm[..., :3] / nrm[..., :3].norm(dim=-1, keepdim=True)
    k = {0: 6.0, 1: 4.0, 2: 1.0}
    luma = torch.tensor([0.299, 0.587, 0.114], dtype=torch.float64, device="cuda")
    ys, xs = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    for it in range(min(max(case["iterations"], 1), 7)):
        c = rad[..., :3]
        lum = (c * luma).sum(-1)
        acc, ws = torch.zeros_like(c), torch.zeros_like(lum)
        for ty in range(-2, 3):
            iy = (ys + ty * (1 << it)).clamp(0, h - 1)
            for tx in range(-2, 3):
                ix = (xs + tx * (1 << it)).clamp(0, w - 1)

                def at(v):
                    return v[iy][:, ix]
                wt = k[abs(tx)] * k[abs(ty)] / 256.0 * torch.exp(-(at(p) - p).square().sum(-1) / sp2)
                wt = wt * torch.exp(-(1.0 - (at(n) * n).sum(-1)).clamp(min=0) / sn2)
                wt = wt * torch.exp(-(at(lum) - lum).square() / sl2)
                wt = torch.where(at(miss), torch.zeros_like(wt), wt)
                acc += at(c) * wt[..., None]
                ws += wt
        out = torch.where((miss | ~(ws > 0))[..., None], c, acc / ws[..., None])
        rad = torch.cat([out, rad[..., 3:]], -1)
    return rad


def _exact_network(params, pos, nrm, wo):
    """The network's mixture, its weights rounded to bfloat16 as they are kept for the
    tensor cores (biases are not), its arithmetic in 64 bits."""
    x = ((pos + BOUNDS) / (2.0 * BOUNDS)).clamp(0.0, 1.0)
    f = math.pi * 2.0 ** torch.arange(12, dtype=torch.float64, device="cuda")
    cols = []
    for a in range(3):
        cols += [torch.sin(x[:, a:a + 1] * f), torch.cos(x[:, a:a + 1] * f)]
    y = torch.cat(cols + [nrm, wo, torch.zeros((len(x), 2), dtype=torch.float64, device="cuda")], 1)
    at = 0
    for layer, (i, o) in enumerate(_layers()):
        wt, b = params[at:at + o * i].view(o, i), params[at + o * i:at + o * i + o]
        at += o * i + o
        y = y @ wt.T + b
        if layer < 4:
            y = torch.relu(y)
    r = y[:, :40].reshape(-1, 8, 5)
    mu = r[:, :, :3] / r[:, :, :3].norm(dim=2, keepdim=True).clamp(min=1e-6)
    kappa = (torch.nn.functional.softplus(r[:, :, 3]) + 0.1).clamp(max=1000.0)
    return mu, kappa, torch.softmax(r[:, :, 4], 1)


def _rounded(params):
    p, at = params.clone(), 0
    for i, o in _layers():
        p[at:at + o * i] = p[at:at + o * i].float().bfloat16().double()
        at += o * i + o
    return p


def exact(case, seed):
    if case["op"] == "atrous":
        return _exact_atrous(case, seed)
    if case["op"] not in ("train", "eval"):
        return None     # paths: one rounding apart, a path takes another way
    n = case["samples"] if case["op"] == "train" else case["points"]
    params, s = _mlp_inputs(n, seed)
    params = torch.from_numpy(params).cuda().double()
    s = torch.from_numpy(s).cuda().double()
    pos, w, om, nrm, wo = s[:, 0:3], s[:, 3], s[:, 4:7], s[:, 8:11], s[:, 12:15]
    if case["op"] == "eval":
        mu, kappa, pi = _exact_network(_rounded(params), pos, nrm, wo)
        return torch.cat([torch.cat([mu, kappa[..., None]], 2), pi.view(-1, 2, 4)], 1)
    p = _rounded(params).requires_grad_(True)
    mu, kappa, pi = _exact_network(p, pos, nrm, wo)
    cosw = (mu * om[:, None]).sum(2)
    lq = pi.clamp(min=1e-30).log() + kappa.log() - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa))
    nll = -torch.logsumexp(lq + kappa * (cosw - 1.0), 1)
    w = torch.minimum(w, 20.0 * w.mean())
    grad, = torch.autograd.grad((w / w.sum() * nll).sum(), p)
    # the first Adam step: both moments are the gradient's own
    stepped = params - 1e-2 * grad / (grad.abs() + 1e-8)
    return {"params": stepped, "grad": 1024.0 * grad}
