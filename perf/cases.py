"""The performance cases: what a renderer asks of the compute stage, call by call.

A case is a plain dict; `prepare` makes what a program has in hand before the
call (a context with its volumes, the previous frames, the uniform blocks),
`run` makes one pass through the public entry points, `work` says what the
pass cannot do without and `exact` evaluates the same pass in FP64 with plain
torch.  Kinds:

  frame   one frame of a view session: 1 pixel per 4x4 block marched, the
          rest reprojected, TXAA resolved (Context.render_frame)
  passes  the same frame with the reference's constants, one call per pass
          as the reference records them: render, txaa, tonemap
  full    a frame with every pixel marched (a session's first frame, a still)
  batch   many views in one call (Context.render_batch): stills of uneven
          size, or the checkerboard frames a server owes its sessions
  post    god rays and tone map over a finished frame
  seeded  a scene change: the volumes generated from a new seed, then the
          first frame (small, so the change itself is what counts)
  assets  a scene load: the volumes decoded from TGA slice stacks, the 2D maps
          uploaded, then the first frame

Sizes are those of the benchmark's configurations (640x360, 1280x720,
1920x1080 sessions; 960x540 and 3840x2160 stills; the batch's five sizes) and
odd ones beside them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from meteoros_gb300 import abi, scenes
from meteoros_gb300.renderer import Context, FrameInputs, Session

# The batched views' sizes, and the sizes sessions are served at.
STILL_SIZES = scenes.CONFIG3_RESOLUTIONS
SESSION_SIZES = ((640, 360), (1280, 720), (640, 360), (1920, 1080))
LIGHT = (1.0, 1.0, 0.57, 1.0)  # SunAndSky.lightColor


def _case(name, kind, width, height, storage="rgba8", **more):
    return dict({"name": name, "kind": kind, "width": width, "height": height, "storage": storage}, **more)


def listed():
    return [
        # A session's steady frame at the commonest streamed size: 14 400 rays, launch latency counts.
        _case("frame_360p", "frame", 640, 360),
        # The headline workload.
        _case("frame_1080p", "frame", 1920, 1080),
        # The same at 4K, where the checkerboard alone is half a million rays.
        _case("frame_4k", "frame", 3840, 2160),
        # A resizable window's size through the reference's constants and its separate passes.
        _case("passes_ragged", "passes", 1366, 769),
        # A session's first frame: every pixel marched.
        _case("full_540p", "full", 960, 540),
        # The precision form's stills: FP16 volumes and FP64 shells at 4K, bfloat16 at an odd size.
        _case("full_4k_fp16", "full", 3840, 2160, "fp16"),
        _case("full_ragged_bf16", "full", 1603, 901, "bf16"),
        # Offline batches of stills with their own weather maps and step budgets.
        _case("batch_stills", "batch", 0, 0, views=20, checkerboard=False),
        # What a serving loop launches: one checkerboard frame of each of its sessions.
        _case("batch_sessions", "batch", 0, 0, views=24, checkerboard=True),
        # The passes after the compute stage.
        _case("post_1080p", "post", 1920, 1080, ldr="rgba8"),
        # A scene change from a seed, and the load of a scene from its asset files.
        _case("scene_seeded", "seeded", 320, 180),
        _case("scene_assets", "assets", 320, 180),
    ]


def draw(rng):
    """One more case of the same ranges (rng: random.Random)."""
    kind = rng.choice(("frame", "frame", "frame", "passes", "full", "full", "batch", "post", "seeded", "assets"))
    storage = rng.choice(("rgba8", "rgba8", "fp16", "bf16"))
    if kind == "batch":
        checkerboard = rng.random() < 0.5
        return {"kind": kind, "width": 0, "height": 0, "storage": storage, "checkerboard": checkerboard,
                "views": rng.randint(2, 24 if checkerboard else 14), "first": rng.randint(0, 4)}
    if kind in ("seeded", "assets"):
        w = rng.randint(96, 640)
        return {"kind": kind, "width": w, "height": max(36, int(w * rng.uniform(0.4, 1.0))), "storage": storage}
    lo, hi = (160.0, 3840.0) if kind != "full" else (200.0, 2400.0)
    w = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    h = max(64, int(w * rng.uniform(0.42, 0.7)))
    out = {"kind": kind, "width": w, "height": h, "storage": storage}
    if kind in ("passes", "post"):
        out["storage"] = "rgba8"
        out["ldr"] = rng.choice(("rgba8", "rgba32f"))
    return out


# ---------------------------------------------------------------------------
# State
# ---------------------------------------------------------------------------
STORAGE = {"rgba8": abi.MT_STORAGE_U8, "fp16": abi.MT_STORAGE_F16, "bf16": abi.MT_STORAGE_BF16}


def _image(h, w, channels=4, dtype=torch.float32):
    shape = (h, w, channels) if channels > 1 else (h, w)
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _with_storage(params, storage):
    p = scenes.C_copy(abi.Params(), params)
    p.storage = STORAGE[storage]
    p.fp64_shells = 0 if storage == "rgba8" else 1
    return p


def _frame_pair(seed, w, h, storage, reference=False):
    """Two consecutive frames of a seeded session: [(camera, camera_old, time, params)] * 2."""
    k = 1 + seed % 15  # the slot of the second frame
    if reference:
        pitch, t = 2.0 + (seed * 7 % 23), 0.16 * (seed % 50)
        cams = [scenes.look((0.0, 0.0, 2.0), yaw, pitch, 45.0, w, h) for yaw in (0.0, 0.5)]
        params = abi.params_reference()
        out = []
        for i in (0, 1):
            tm = abi.time_init()
            tm.frame_count_mod16 = k - 1 + i
            tm.time[0], tm.time[1] = 0.16, t + 0.16 * i
            out.append((cams[i], cams[0], tm, params))
        return out
    seq = scenes.config_sequence(seed, w, h, frames=k + 1)[k - 1:]
    return [(cam, old, tm, _with_storage(params, storage)) for cam, old, tm, params in seq]


def _asset_files(vols):
    """TGA slice stacks as the reference ships them: 32-bit run-length files,
    bottom row first, one literal packet a row."""
    stacks = []
    for vol in (vols["base"], vols["detail"]):
        n = vol.shape[0]
        head = bytes([0, 0, 10, 0, 0, 0, 0, 0, 0, 0, 0, 0, n & 255, n >> 8, n & 255, n >> 8, 32, 8])
        rows = np.empty((n, n, 1 + 4 * n), np.uint8)
        rows[..., 0] = n - 1
        rows[..., 1:] = vol[:, ::-1][..., [2, 1, 0, 3]].reshape(n, n, 4 * n)
        files = [head + rows[z].tobytes() for z in range(n)]
        stacks.append(((C.c_void_p * n)(*[C.cast(C.c_char_p(f), C.c_void_p) for f in files]),
                       (C.c_size_t * n)(*[len(f) for f in files]), n, files))
    return stacks


def prepare(case, seed):
    kind, w, h, storage = case["kind"], case["width"], case["height"], case["storage"]
    ctx = Context(0)
    ctx.generate_volumes(seed)
    s = {"kind": kind, "ctx": ctx}
    if kind in ("frame", "passes"):
        first, f = _frame_pair(seed, w, h, storage, kind == "passes")
        session = Session(ctx, w, h)
        session.frame(FrameInputs(*first))
        s.update(f=f, prev=session.raw[0], cur=session.raw[1], hist=session.resolved[0], out=session.resolved[1],
                 mask=session.masks[1], ldr=_ldr_image(case, h, w) if kind == "passes" else None)
    elif kind in ("full", "seeded", "assets"):
        cam, tm, params, _ = scenes.config_view(seed, w, h)
        s.update(f=(cam, cam, tm, _with_storage(params, storage)), cur=_image(h, w), mask=_image(h, w, 1))
        if kind == "seeded":
            s["seed"] = seed + 1
        elif kind == "assets":
            # the scene to load: what a generator with another seed gives, as files and arrays on the host
            ctx.generate_volumes(seed + 1)
            s["vols"] = ctx.download_volumes()
            s["stacks"] = _asset_files(s["vols"])
            ctx.generate_volumes(seed)
    elif kind == "batch":
        s["views"], s["images"] = _batch(ctx, case, seed)
    elif kind == "post":
        cam, tm, params, _ = scenes.config_view(seed, w, h)
        s.update(inp=_image(h, w), mask=_image(h, w, 1), lit=_image(h, w), ldr=_ldr_image(case, h, w))
        ctx.render(cam, cam, tm, params, None, s["inp"], s["mask"], abi.MT_RENDER_FULL)
        tm.time[1] = 0.16 * (seed % 1000)
        # the pass blurs toward a static sun: seen by a camera that looks its way
        s["f"] = (scenes.look((0.0, 0.0, 2.0), seed % 7, 5.0 + seed % 20, 45.0, w, h), cam, tm, params)
    return s


def _ldr_image(case, h, w):
    return _image(h, w, 4, torch.float32 if case.get("ldr") == "rgba32f" else torch.uint8)


def _batch(ctx, case, seed):
    n, first, checkerboard = case["views"], case.get("first", 0), case["checkerboard"]
    rng = np.random.default_rng(seed)
    views, images = [], []
    for v in range(n):
        if checkerboard:
            w, h = SESSION_SIZES[(v + first) % len(SESSION_SIZES)]
            start, (cam, old, tm, params) = _frame_pair(seed * 100 + v, w, h, case["storage"])
            prev = _image(h, w)
            ctx.render(start[0], start[0], start[2], params, None, prev, None, abi.MT_RENDER_FULL)
        else:
            w, h = STILL_SIZES[(v + first) % len(STILL_SIZES)]
            cam, tm, params, _ = scenes.config_view(seed * 1000 + v, w, h, steps=int(rng.integers(64, 129)))
            params = _with_storage(params, case["storage"])
            params.weather_slot = v
            if v:
                ctx.generate_weather(v, seed + v)
            old, prev = cam, None
        cur, mask = _image(h, w), _image(h, w, 1)
        images.append((prev, cur, mask))
        views.append(scenes.make_view(cam, old, tm, params, cur, prev, mask,
                                      abi.MT_RENDER_CHECKERBOARD if checkerboard else abi.MT_RENDER_FULL))
    return views, images


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "batch":
        ctx.render_batch(s["views"])
        return [(cur, mask) for _, cur, mask in s["images"]]
    cam, old, tm, params = s["f"]
    if kind == "frame":
        ctx.render_frame(cam, old, tm, params, s["prev"], s["cur"], s["hist"], s["out"], s["mask"])
        return s["cur"], s["out"], s["mask"]
    if kind == "passes":
        ctx.render(cam, old, tm, params, s["prev"], s["cur"], s["mask"])
        ctx.txaa(cam, old, tm, params, s["cur"], s["hist"], s["out"])
        ctx.tonemap(tm, s["out"], s["ldr"], _ldr_format(s["ldr"]))
        return s["cur"], s["out"], s["mask"], s["ldr"]
    if kind == "post":
        ctx.godrays(cam, LIGHT, s["mask"], s["inp"], s["lit"])
        ctx.tonemap(tm, s["lit"], s["ldr"], _ldr_format(s["ldr"]))
        return s["lit"], s["ldr"]
    if kind == "seeded":
        ctx.generate_volumes(s["seed"])
    elif kind == "assets":
        for volume, (files, sizes, n, _) in zip((abi.MT_VOLUME_BASE, abi.MT_VOLUME_DETAIL), s["stacks"]):
            status = ctx.lib.mt_decode_tga_volume(ctx.handle, volume, files, sizes, n,
                                                  torch.cuda.current_stream().cuda_stream)
            if status != abi.MT_OK:
                raise abi.MeteorosError(status, ctx.lib.mt_last_error(ctx.handle).decode())
        ctx.upload_volumes(curl=s["vols"]["curl"], weather=s["vols"]["weather"])
    ctx.render(cam, old, tm, params, None, s["cur"], s["mask"], abi.MT_RENDER_FULL)
    return s["cur"], s["mask"]


def _ldr_format(ldr):
    return abi.MT_LDR_RGBA8 if ldr.dtype == torch.uint8 else abi.MT_LDR_RGBA32F


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
# FP32 operations of the raymarch by visited pixel, marching ray, primary
# sample and light sample, and the mean samples of a ray over seeded views:
# (marching rays per pixel, primary samples and in-cloud steps per ray) with
# the benchmark's parameters (a budget of 128 steps) and with the reference's.
FLOPS_PIXEL, FLOPS_RAY, FLOPS_PRIMARY, FLOPS_LIGHT = 132.6, 506.5, 307.8, 229.6
MEAN_CONFIG, MEAN_REFERENCE = (0.83, 33.0, 15.5), (0.83, 17.0, 17.0)
VOLUME_BYTES = 4 * (128 ** 3 + 32 ** 3 + 128 ** 2 + 512 ** 2)
REPROJECT_FLOPS, TXAA_FLOPS, GODRAY_FLOPS, TONEMAP_FLOPS = 170.0, 330.0, 100 * 26.0, 120.0
GENERATE_FLOPS = 9 * 27 * 12.0 + 4 * 90.0  # a base texel: nine Worley octaves, four of gradient noise


def _march_flops(pixels, mean=MEAN_CONFIG):
    rays, steps, cloud = mean
    return pixels * (FLOPS_PIXEL + rays * (FLOPS_RAY + steps * FLOPS_PRIMARY + cloud * 6 * FLOPS_LIGHT))


def work(case):
    kind, w, h = case["kind"], case["width"], case["height"]
    px = w * h
    volumes = VOLUME_BYTES * (1 if case["storage"] == "rgba8" else 2)
    ldr = px * (16 if case.get("ldr") == "rgba32f" else 4)
    if kind == "frame":  # previous frame and history read, frame and result written, 1/16 of the mask
        return {"bytes": volumes + px * (4 * 16 + 4 / 16),
                "flops": _march_flops(px / 16) + px * (REPROJECT_FLOPS + TXAA_FLOPS)}
    if kind == "passes":
        return {"bytes": volumes + px * (4 * 16 + 4 / 16) + ldr,
                "flops": _march_flops(px / 16, MEAN_REFERENCE) + px * (REPROJECT_FLOPS + TXAA_FLOPS + TONEMAP_FLOPS)}
    if kind == "full":
        return {"bytes": volumes + px * 20, "flops": _march_flops(px)}
    if kind == "post":
        return {"bytes": px * (16 + 4 + 16) + ldr, "flops": px * (GODRAY_FLOPS + TONEMAP_FLOPS)}
    if kind == "seeded":  # the volumes in the three storages written, the frame
        return {"bytes": VOLUME_BYTES * 5 + px * 20, "flops": _march_flops(px) + 128 ** 3 * GENERATE_FLOPS}
    if kind == "assets":  # the files read, the volumes in the three storages written, the frame
        return {"bytes": VOLUME_BYTES * 6 + px * 20, "flops": _march_flops(px)}
    sizes = SESSION_SIZES if case["checkerboard"] else STILL_SIZES
    total = sum(a * b for a, b in (sizes[(v + case.get("first", 0)) % len(sizes)] for v in range(case["views"])))
    if case["checkerboard"]:
        return {"bytes": volumes + total * (2 * 16 + 4 / 16),
                "flops": _march_flops(total / 16) + total * REPROJECT_FLOPS}
    # a budget of 64 to 128 steps: three quarters of the samples
    return {"bytes": volumes + total * 20, "flops": 0.75 * _march_flops(total)}


# ---------------------------------------------------------------------------
# The same pass in FP64, in plain torch.  The march has hard thresholds (a step
# in or out of cloud, the early exit, the jitter index taken from int(t)): where
# FP32 falls on the other side than FP64 a pixel moves by a step's contribution,
# which is most of the FP32 results' distance from these.  The god-ray mask has
# no such value (None): it is 0 wherever a ray ended opaque, and what is not is
# the fraction of a number around 1 in steps of the accumulated density, so
# those flips are all there is to compare.  Nor have the tone map's bytes.
# ---------------------------------------------------------------------------
F64 = torch.float64


def exact(case, seed):
    s = prepare(case, seed)
    kind, ctx, w, h = s["kind"], s["ctx"], case["width"], case["height"]
    if kind == "batch":
        out = []
        for view, (prev, _, _) in zip(s["views"], s["images"]):
            vols = _volumes(ctx, case["storage"], view.params.weather_slot)
            f = (view.camera, view.camera_old, view.time, view.params)
            out.append((_render64(vols, f, prev, view.width, view.height), None))
        return out
    if kind == "post":
        lit = _godrays64(s["f"][0], s["mask"].to(F64), s["inp"].to(F64), w, h)
        return lit, None if s["ldr"].dtype == torch.uint8 else _tonemap64(s["f"][2], lit, w, h)
    if kind == "seeded":
        ctx.generate_volumes(s["seed"])  # bytes, the same on every machine: the frame's input
    if kind == "assets":
        ctx.upload_volumes(**s["vols"])
    cur = _render64(_volumes(ctx, case["storage"], 0), s["f"], s.get("prev"), w, h)
    if kind not in ("frame", "passes"):
        return cur, None
    out = _txaa64(s["f"], cur, s["hist"].to(F64), w, h)
    if kind == "frame":
        return cur, out, None
    return cur, out, None, None if s["ldr"].dtype == torch.uint8 else _tonemap64(s["f"][2], out, w, h)


def _t(x):
    return torch.tensor([float(v) for v in x], dtype=F64, device="cuda")


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _mix(x, y, a):
    return x * (1.0 - a) + y * a


def _volumes(ctx, storage, slot):
    """{name: (texels on an axis, (texels, 4) values)} of what the storage holds."""
    if storage == "rgba8":
        vols = {k: v.astype(np.float64) / 255.0 for k, v in ctx.download_volumes(slot).items()}
    else:
        bits = ctx.download_volumes_16(STORAGE[storage], slot)
        if storage == "fp16":
            vols = {k: v.view(np.float16).astype(np.float64) for k, v in bits.items()}
        else:
            vols = {k: (v.astype(np.uint32) << 16).view(np.float32).astype(np.float64) for k, v in bits.items()}
    return {k: (v.shape[0], torch.from_numpy(v.reshape(-1, 4)).cuda()) for k, v in vols.items()}


def _sample(volume, *coords):
    """LINEAR filter, REPEAT, over the axes given (x fastest)."""
    n, texels = volume
    cells = []
    for c in coords:
        u = c * n - 0.5
        i = torch.floor(u)
        i0 = i.to(torch.int64)
        cells.append(((i0 % n, (i0 + 1) % n), (u - i)[:, None]))

    def value(axis, offset):
        (i0, i1), a = cells[axis]
        lo, hi = offset + i0 * n ** axis, offset + i1 * n ** axis
        if axis == 0:
            p, q = texels[lo], texels[hi]
        else:
            p, q = value(axis - 1, lo), value(axis - 1, hi)
        return p + a * (q - p)

    return value(len(coords) - 1, torch.zeros_like(cells[0][0][0]))


def _jitter(tm, index, repro=False):
    """The (x, y) jitter of slot `index` (a tensor or an int), before its scale."""
    i = torch.as_tensor(index, device="cuda") // 2
    h1, h2 = _t(tm.halton_seq1), _t(tm.halton_seq2)
    h3, h4 = (h1, h2) if repro else (_t(tm.halton_seq3), _t(tm.halton_seq4))
    return torch.cat([h1, h3])[i], torch.cat([h2, h4])[i]


def _eye(cam, p):
    return p.eye_sign * _t(cam.eye)[:3]


def _rays(cam, tm, p, ux, uy, w, h, repro=False):
    v = _t(cam.view).reshape(4, 4)  # v[c][r]
    right, up, look = _unit(v[:3, 0]), _unit(v[:3, 1]), -_unit(v[:3, 2])
    jx, jy = _jitter(tm, tm.frame_count_mod16, repro)
    nx, ny = ux * 2.0 - 1.0 + jx / w, uy * 2.0 - 1.0 + jy / h
    return _unit(look + (nx * cam.tan_fov_by_2[0])[:, None] * right + (ny * cam.tan_fov_by_2[1])[:, None] * up)


def _sphere(eye, d, centre, radius):
    """(point, t): t is the distance from the normalised origin, as the shader has it."""
    o = (eye - centre) / radius
    b, c = 2.0 * _dot(d, o), _dot(o, o) - 1.0
    a = _dot(d, d)
    root = torch.sqrt(torch.clamp(b * b - 4.0 * a * c, min=0.0))
    t = (-b - root) / (2.0 * a)
    t = torch.where(t < 0.0, (-b + root) / (2.0 * a), t)
    point = (o + t[:, None] * d) * radius + centre
    return point, (point - o).norm(dim=-1)


def _hg(c, e):
    return (1.0 - e * e) / (1.0 + e * e - 2.0 * e * c) ** 1.5 * 0.07957747154594767


def _smooth(lo, hi, x):
    t = torch.clamp((x - lo) / (hi - lo), 0.0, 1.0)
    return t * t * (3.0 - 2.0 * t)


def _sky(p, eye, d):
    sun = _t(p.sky_sun_pos)
    sun_dir = _unit(sun - eye)
    zen = torch.clamp(_unit(sun)[1], -1.0, 1.0)
    sun_e = 0.780 * 1000.0 * torch.clamp(1.0 - 2.718281828459 ** (-((1.6110731557 - torch.acos(zen)) / 1.5)), min=0.0)
    fade = 1.0 - torch.clamp(1.0 - torch.exp(sun[1] / 450000.0), 0.0, 1.0)
    beta_r = _t((5.804542996261093e-6, 1.3562911419845635e-5, 3.0265902468824876e-5)) * (1.0 + fade)
    beta_m = 0.434 * (0.2 * 10.0 * 10e-18) * _t((1.839991851443397, 2.779802391966052, 4.079047954386109)) * 0.005
    zenith = torch.acos(torch.clamp(d[:, 1], min=0.0))
    inv = 1.0 / (torch.cos(zenith) + 0.15 * (93.885 - zenith * 180.0 / 3.14159265) ** -1.253)
    fex = torch.exp(-beta_r * (8.4e3 * inv)[:, None] + beta_m * (1.25e3 * inv)[:, None])
    cos_t = _dot(sun_dir, d)
    phase_r = 0.05968310365946075 * (1.0 + (cos_t * 0.5 + 0.5) ** 2)
    betas = (beta_r * phase_r[:, None] + beta_m * _hg(cos_t, 0.8)[:, None]) / (beta_r + beta_m)
    lin = (sun_e * betas * (1.0 - fex)) ** 1.5
    y = 1.0 - sun_dir[1]
    lin = lin * _mix(torch.ones_like(lin), (sun_e * betas * fex) ** 0.5, torch.clamp(y ** 5, 0.0, 1.0))
    edge = 0.999956676946448443553574619906976478926848692873900859324
    l0 = 0.1 * fex + sun_e * 15000.0 * fex * _smooth(edge, edge + 0.00002, cos_t)[:, None]
    return (lin + l0) * 0.04 + _t((0.0, 0.0003, 0.00075))


def _height_gradient(h, kind):
    h = torch.clamp(h, 0.0, 1.0)
    strato = torch.clamp(h / 0.25 * (1.0 - (h - 0.3) / 0.35), min=0.0)
    stratus = torch.clamp(h / 0.1 * (1.0 - (h - 0.2) / 0.1), min=0.0)
    a = _mix(stratus, strato, torch.clamp(kind * 2.0, 0.0, 1.0))
    b = _mix(strato, stratus, torch.clamp((kind - 0.5) * 2.0, 0.0, 1.0))
    return _mix(a, b, kind)


def _density(p, vols, point, lo, mul, gradient):
    n = _sample(vols["base"], point[:, 0], point[:, 1], point[:, 2])
    fbm = torch.clamp(n[:, 1] * 0.625 + n[:, 2] * 0.25 + n[:, 3] * 0.125, 0.0, 1.0)
    shape = torch.clamp((n[:, 0] - (fbm - 0.9)) / (1.0 - (fbm - 0.9)), 0.0, 1.0) * gradient
    return torch.clamp((torch.minimum(torch.maximum(shape, lo), torch.ones_like(lo)) - lo) / (1.0 - lo), 0.0, 1.0) * mul


def _light_energy(h, dl, ds, phase, cos_angle):
    primary = torch.exp(-dl)
    att = torch.maximum(primary + (cos_angle - 0.7) / 0.3 * (primary * 0.25 - primary), primary)
    depth = 0.05 + ds ** torch.clamp(0.5 + (h * 0.125 - 0.3) / 0.55 * 1.5, 0.5, 2.0)
    vert = torch.clamp(0.1 + (h * 1.5 - 0.07) / 0.27 * 0.9, 0.1, 1.0) ** 0.8
    return att * primary * depth * vert * phase * 5.0


CONE = ((0.1, 0.25, -0.15), (0.2, 0.5, 0.2), (-0.2, 0.1, -0.1), (-0.05, 0.75, 0.05), (-0.1, 1.0, 0.0), (0.0, 3.0, 0.0))


def _cone(light):
    k = int(torch.argmax(light.abs()))
    major = torch.zeros_like(light)
    major[k] = light.abs()[k]
    z = torch.linalg.cross(light, major)
    x = torch.linalg.cross(z, light)
    return [x * a + light * b + z * c for a, b, c in CONE]


def _march64(vols, cam, tm, p, d):
    """Colour and opacity of the rays d (n, 3) from the eye, all above the fade elevation."""
    eye = _eye(cam, p)
    centre = eye.clone()
    centre[1] = -p.earth_radius
    thick = p.shell_outer_radius - p.shell_inner_radius
    base = centre.clone()
    base[1] = p.shell_inner_radius - p.earth_radius
    start, t0 = _sphere(eye, d, centre, p.shell_inner_radius)
    _, t1 = _sphere(eye, d, centre, p.shell_outer_radius)
    steps = torch.floor(_mix(float(p.steps_min), float(p.steps_max), 1.0 - d[:, 1]))
    if p.steps_min == p.steps_max:
        steps = torch.full_like(steps, p.steps_min)
    step = (t1 - t0) / steps
    light = _unit(_t(p.sun_light_pos) - eye)
    cos_a = _dot(d, light)
    phase = torch.maximum(_hg(cos_a, 0.6), 0.7 * _hg(cos_a, 0.89))
    cone = _cone(light)
    len_in = (start - eye).norm(dim=-1)
    wind = _t(p.wind_dir) * p.wind_speed * tm.time[1]
    skew = _t(p.skew_dir) * p.cloud_top_offset * 0.009
    t, accum, trans, colour = t0.clone(), torch.zeros_like(t0), torch.ones_like(t0), torch.zeros_like(t0)
    alive = torch.nonzero(t < t1)[:, 0]
    for _ in range(2 * max(p.steps_min, p.steps_max) + 8):
        if not alive.numel():
            break
        dd, tt = d[alive], t[alive]
        slot = (tm.frame_count_mod16 + tt.to(torch.int64)) % 16
        jx, jy = (j / 75.0 for j in _jitter(tm, slot))
        pos = eye + tt[:, None] * (dd + torch.stack([jx, (jx + jy) * 1.18, jy], -1))
        up = _unit(pos - centre)
        h = (_dot(dd, up) * ((pos - eye).norm(dim=-1) - len_in[alive])).abs() / thick
        point = (pos - base) / thick / p.noise_period + h[:, None] * skew + wind
        if p.coverage_mode == 1:
            wd = _sample(vols["weather"], (pos[:, 0] - centre[0]) / p.weather_scale,
                         (pos[:, 2] - centre[2]) / p.weather_scale)
            lo, mul, kind = 1.0 - wd[:, 0], wd[:, 0], wd[:, 2]
        else:
            lo = mul = torch.full_like(h, p.coverage)
            kind = torch.zeros_like(h)
        grad = _height_gradient(h, kind) if p.height_gradient else torch.ones_like(h)
        ds = torch.zeros_like(h)
        may = torch.nonzero((grad > lo) & (mul > 0.0))[:, 0]  # elsewhere the density is 0 whatever the shape
        ds[may] = _density(p, vols, point[may], lo[may], mul[may], grad[may]) * 0.380
        k = torch.nonzero(ds > 0.0)[:, 0]
        if k.numel():
            r = alive[k]
            pt, hk, dk = point[k].clone(), h[k], ds[k]
            curl = _sample(vols["curl"], pt[:, 0], pt[:, 1])
            pt[:, :2] += curl[:, :2] * (1.0 - hk)[:, None] * 0.5
            hf = _sample(vols["detail"], pt[:, 0], pt[:, 1], pt[:, 2])
            fbm = hf[:, 0] * 0.625 + hf[:, 1] * 0.25 + hf[:, 2] * 0.125
            edge = torch.clamp(_mix(fbm, 1.0 - fbm, torch.clamp(hk * 2.0, 0.0, 1.0)), 0.0, 1.0) * 0.005
            accum[r] += (dk * 1.4 - edge) / (1.0 - edge) * 0.5
            dl = torch.zeros_like(dk)
            for i, c in enumerate(cone):
                at = (pos[k] + (step[r] * i)[:, None] * c - base) / thick
                cbl = _density(p, vols, at, lo[k], mul[k], grad[k])
                dl += torch.where(cbl > 0.0, (1.5 * cbl - edge) / (1.0 - edge), torch.zeros_like(cbl))
            e = _light_energy(hk, dl, dk, phase[r], cos_a[r])
            trans[r] = _mix(trans[r], e, 1.0 - accum[r])
            colour[r] += trans[r]
        done = accum[alive] >= p.accum_limit
        accum[alive[done]] = 1.0
        t[alive] += step[alive]
        alive = alive[~done & (t[alive] < t1[alive])]
    return colour, accum * _smooth(0.0, 1.0, torch.clamp((d[:, 1] - 0.06) / 0.14, max=1.0))


def _pixels64(vols, cam, tm, p, w, h, xs, ys):
    d = _rays(cam, tm, p, xs / w, 1.0 - ys / h, w, h)
    elevation = d[:, 1:2]
    below = _mix(_t((0.0, 0.064, 0.204)), _t((0.0, 0.365, 0.475)), -elevation * 5.5)
    rgb = torch.where(elevation < 0.0, below, _sky(p, _eye(cam, p), d) * torch.clamp(elevation, min=0.620))
    for k in torch.nonzero(d[:, 1] >= 0.06)[:, 0].split(1 << 20):
        colour, opacity = _march64(vols, cam, tm, p, d[k])
        rgb[k] = _mix(rgb[k], colour[:, None], opacity[:, None])
    return torch.cat([rgb, torch.ones_like(xs)[:, None]], 1)


def _grid(w, h):
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    return x.reshape(-1).to(F64), y.reshape(-1).to(F64)


def _old_uv(f, x, y, w, h, repro):
    cam, old, tm, p = f
    eye = _eye(cam, p)
    centre = eye.clone()
    centre[1] = -p.earth_radius
    point, _ = _sphere(eye, _rays(cam, tm, p, x, y, w, h, repro), centre, p.shell_inner_radius)
    v = _t(old.view).reshape(4, 4)
    o = point @ v[:3, :3] + v[3, :3]
    o = o / -o[:, 2:3]
    return o[:, 0] / cam.tan_fov_by_2[0] * 0.5 + 0.5, o[:, 1] / cam.tan_fov_by_2[1] * 0.5 + 0.5


def _half_away(x):
    return torch.sign(x) * torch.floor(x.abs() + 0.5)


def _render64(vols, f, prev, w, h):
    cam, _, tm, p = f
    x, y = _grid(w, h)
    if prev is None:  # every pixel marched
        return _pixels64(vols, cam, tm, p, w, h, x, y).reshape(h, w, 4)
    ux, uy = x / w, y / h
    ou, ov = _old_uv(f, ux, uy, w, h, True)
    flat, cur = prev.to(F64).reshape(-1, 4), torch.zeros((w * h, 4), dtype=F64, device="cuda")
    for i in range(10):
        ix = torch.clamp(_half_away((ou - (ou - ux) * (i / 10.0)) * w), 0, w - 1).to(torch.int64)
        iy = torch.clamp(_half_away((ov - (ov - uy) * (i / 10.0)) * h), 0, h - 1).to(torch.int64)
        cur += flat[iy * w + ix]
    cur /= 10.0
    # one pixel per 4x4 block, over the 32-block groups the reference dispatches
    sx, sy = p.slot_x[tm.frame_count_mod16], p.slot_y[tm.frame_count_mod16]
    groups = [32 * ((n // 4 + 31) // 32) for n in (w, h)]
    mine = (x >= sx) & (y >= sy) & ((x - sx) % 4 == 0) & ((y - sy) % 4 == 0)
    mine &= ((x - sx) / 4 < groups[0]) & ((y - sy) / 4 < groups[1])
    k = torch.nonzero(mine)[:, 0]
    cur[k] = _pixels64(vols, cam, tm, p, w, h, x[k], y[k])
    return cur.reshape(h, w, 4)


def _border(img, x, y, w, h):
    """LINEAR filter, CLAMP_TO_BORDER with opaque black, over a (h, w, 4) image."""
    pad = torch.zeros((h + 2, w + 2, 4), dtype=F64, device="cuda")
    pad[..., 3] = 1.0
    pad[1:-1, 1:-1] = img
    u, v = x * w - 0.5, y * h - 0.5
    i, j = torch.floor(u), torch.floor(v)
    a, b = (u - i)[:, None], (v - j)[:, None]

    def at(ii, jj):
        return pad[torch.clamp(jj + 1, 0, h + 1).to(torch.int64), torch.clamp(ii + 1, 0, w + 1).to(torch.int64)]

    top = at(i, j) + a * (at(i + 1, j) - at(i, j))
    low = at(i, j + 1) + a * (at(i + 1, j + 1) - at(i, j + 1))
    return top + b * (low - top)


def _landing(n):
    """The pixel each fragment of an axis stores to: an integer the shader takes from FP32 arithmetic."""
    f = np.arange(n, dtype=np.float32)
    q = np.float32(n) * ((f + np.float32(0.5)) / np.float32(n))
    return np.clip(np.floor(q.astype(np.float64) + 0.5), 0, n - 1).astype(np.int64)


def _txaa64(f, cur, hist, w, h):
    p = f[3]
    x, y = _grid(w, h)
    prev = _border(hist, *_old_uv(f, (x + 0.5) / w, (y + 0.5) / h, w, h, False), w, h)
    lx, ly = (torch.from_numpy(_landing(n)).cuda() for n in (w, h))
    pad = torch.zeros((h + 2, w + 2, 4), dtype=F64, device="cuda")
    pad[1:-1, 1:-1] = cur
    n = torch.stack([pad[ly + 1 + dy][:, lx + 1 + dx].reshape(-1, 4) for dy in (-1, 0, 1) for dx in (-1, 0, 1)])
    cross = n[[1, 3, 4, 5, 7]]
    lo, hi = 0.5 * (n.amin(0) + cross.amin(0)), 0.5 * (n.amax(0) + cross.amax(0))
    avg = 0.5 * (n.mean(0) + cross.mean(0))
    curr = n[4]
    centre = torch.cat([0.5 * (hi + lo)[:, :3], torch.minimum(torch.maximum(avg, lo), hi)[:, 3:]], 1)
    extent = 0.5 * (hi - lo)[:, :3] + 1e-10
    v = prev - centre
    reach = (v[:, :3] / extent).abs().amax(1, keepdim=True)
    prev = torch.where(reach > 1.0, centre + v / reach, prev)
    weights = _t((0.2125, 0.7154, 0.0721))
    l0, l1 = curr[:, :3] @ weights, prev[:, :3] @ weights
    diff = (l0 - l1).abs() / torch.maximum(l0, torch.clamp(l1, min=0.2))
    k = _mix(p.feedback_min, p.feedback_max, (1.0 - diff) ** 2)[:, None]
    return _mix(prev, curr, k).reshape(h, w, 4)


def _fragments(w, h):
    """Per axis, the fragment whose store lands on each pixel (the last one), or -1."""
    out = []
    for n in (w, h):
        frag = np.full(n, -1, np.int64)
        frag[_landing(n)] = np.arange(n)
        out.append(torch.from_numpy(frag).cuda())
    return out


def _godrays64(cam, mask, img, w, h):
    fx, fy = _fragments(w, h)
    sun = _t((0.0, 1.0, 0.0))
    v, proj = _t(cam.view).reshape(4, 4), _t(cam.proj).reshape(4, 4)
    blend = float(_dot(_unit(sun - _t(cam.eye)[:3]), -_unit(v[:3, 2])))
    if blend < 0.0:
        return img
    clip = torch.cat([sun, torch.ones_like(sun[:1])]) @ (v @ proj)
    ssx, ssy = (float(torch.clamp((c + 1.0) / 2.0, 0.0, 1.0)) for c in clip[:2])
    texel = torch.zeros((h, w, 4), dtype=F64, device="cuda")
    texel[..., 0] = mask
    ux = ((fx.to(F64) + 0.5) / w).repeat(h)
    uy = ((fy.to(F64) + 0.5) / h).repeat_interleave(w)
    total = torch.zeros_like(ux)
    for i in range(100):
        s = _border(texel, ux - (ux - ssx) / 100.0 * i, uy - (uy - ssy) / 100.0 * i, w, h)
        total += (s[:, 0] + s[:, 3] / 16581375.0) * 0.001
    out = img.reshape(-1, 4).clone()
    stored = ((fx >= 0).repeat(h) & (fy >= 0).repeat_interleave(w))[:, None]
    add = torch.cat([total[:, None] * _t(LIGHT)[:3], torch.ones_like(total)[:, None]], 1) * blend
    return (out + torch.where(stored, add, torch.zeros_like(add))).reshape(h, w, 4)


def _tonemap64(tm, img, w, h):
    fx, fy = _fragments(w, h)
    c = _border(img, ((fx.to(F64) + 0.5) / w).repeat(h), ((fy.to(F64) + 0.5) / h).repeat_interleave(w), w, h)[:, :3]

    def curve(x):
        return (x * (0.15 * x + 0.05) + 0.004) / (x * (0.15 * x + 0.5) + 0.06) - 0.02 / 0.30

    x, y = _grid(w, h)
    u = 0xFFFFFFFF
    seed = (x.to(torch.int64) * 1664525 + y.to(torch.int64) + int(tm.time[1])) & u
    seed = (seed ^ 61) ^ (seed >> 16)
    seed = (seed * 9) & u
    seed = seed ^ (seed >> 4)
    seed = (seed * 0x27D4EB2D) & u
    seed = seed ^ (seed >> 15)
    noise = seed.to(F64) / 4294967296.0 * 0.01
    white = 1.0 / curve(torch.tensor(100.0, dtype=F64, device="cuda"))
    ldr = torch.cat([(curve(2.5 * c) * white) ** (1.0 / 2.2) + noise[:, None], torch.ones_like(noise)[:, None]], 1)
    stored = ((fx >= 0).repeat(h) & (fy >= 0).repeat_interleave(w))[:, None]
    return torch.where(stored, ldr, torch.zeros_like(ldr)).reshape(h, w, 4)
