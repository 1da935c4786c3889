"""Workloads for timing this library: what a renderer does with it each frame, through the public entry points.

`listed()` names the cases, `draw(rng)` gives others of the same ranges, `prepare` makes what a program holds before
the call (inputs on the device, the handle with its history), `run` is one pass, `work` the bytes and operations the
pass cannot do without, and `exact` the same pass in 64 bits with plain torch.

Sequences come from `tron_grid_gb300.scene` and `fog_scene` (seeded planes with 1-spp noise and exact motion vectors;
seeded froxel volumes).  A temporal case holds a few consecutive frames and walks through them, so that every pass
reprojects the history of the pass before it.
"""
import math

import numpy as np
import torch

import tron_grid_gb300 as tg
from tron_grid_gb300 import fog_scene, scene
from tron_grid_gb300.batch import Batch

WARM = 3  # frames a temporal handle has denoised before the first pass: histories reach the 4-frame fallback limit
STREAM_SIZES = [(160, 90), (320, 180), (640, 360), (1280, 720)]


def listed():
    return [
        # the engine's own chain at the size and in the image formats its published time is for
        dict(name="ref_720p_f16", kind="ref", w=1280, h=720, half=True),
        # the same chain on a 4K display
        dict(name="ref_4k_f16", kind="ref", w=3840, h=2160, half=True),
        # the smallest camera stream (a picture-in-picture or an AI entity's view): launches count
        dict(name="full_160x90_f16", kind="full", w=160, h=90, half=True),
        # the headline: the full filter on a 4K stream, float32 images and state
        dict(name="full_4k_f32", kind="full", w=3840, h=2160, half=False),
        # a resized window, odd in both directions, binary16 state and octahedral normals
        dict(name="full_1917x1077_f16", kind="full", w=1917, h=1077, half=True),
        # a camera cut or a resize: the history is zeroed and every pixel takes the spatial variance estimate
        dict(name="cut_1080p_f32", kind="cut", w=1920, h=1080, half=False),
        # many cameras of uneven sizes in one step (a render farm's or a simulator's streams)
        dict(name="batch_64_f16", kind="batch", n=64, half=True),
        # a program without device buffers of its own: pinned host images in and out
        dict(name="host_1080p_f32", kind="host", w=1920, h=1080, half=False),
        # the engine's froxel grid
        dict(name="fog_320x180x64_f16", kind="fog", w=320, h=180, d=64, half=True),
        # bloom and post-process of a 4K frame into the swapchain image
        dict(name="post_4k_f16", kind="post", w=3840, h=2160, half=True, out="bgra"),
        # the same for a float image kept for later work, at an odd size near the engine's default window
        dict(name="post_1281x721_f32", kind="post", w=1281, h=721, half=False, out="float"),
        # the eye frames of 32 AI entities of mixed resolution, read two ticks behind
        dict(name="eye_32_bgra", kind="eye", n=32, colour="bgra"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame_size(rng, lo, hi):
    """A width spread over its logarithm and a height near 16:9, either of them odd as often as even."""
    w = _log_int(rng, lo, hi)
    h = max(1, min(int(w * rng.uniform(0.5, 0.75)), hi * 9 // 16))
    return w, h


def draw(rng):
    kind = rng.choice(["ref", "ref", "full", "full", "full", "cut", "batch", "host", "fog", "post", "post", "eye"])
    half = rng.random() < 0.5
    if kind in ("ref", "full", "cut"):
        w, h = _frame_size(rng, 96, 1920 if kind == "cut" else 3840)
        return dict(kind=kind, w=w, h=h, half=half)
    if kind == "host":
        w, h = _frame_size(rng, 160, 1920)
        return dict(kind=kind, w=w, h=h, half=half)
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(3, 64), half=half)
    if kind == "fog":
        return dict(kind=kind, w=_log_int(rng, 40, 320), h=_log_int(rng, 24, 180), d=_log_int(rng, 8, 64), half=half)
    if kind == "post":
        w, h = _frame_size(rng, 96, 3840)
        return dict(kind=kind, w=w, h=h, half=half, out=rng.choice(["bgra", "rgba", "float"]))
    return dict(kind="eye", n=rng.randint(2, 32), colour=rng.choice(["bgra", "half", "float"]))


# ------------------------------------------------------------------ inputs ----


def _spec_frames(spec, start, count, half, full):
    """`count` consecutive frames of a plane scene as the handle takes them."""
    sc = scene.PlaneScene(spec, "cuda")
    frames = []
    for t in range(start, start + count):
        f = sc.frame(t)
        fr = dict(radiance=f["radiance"].to(torch.float16) if half else f["radiance"])
        if full:
            fr["depth"] = f["depth"]
            fr["normal"] = scene.oct16_encode(f["normal"]).contiguous() if half else f["normal"]
            fr["motion"] = f["motion"]
        frames.append(fr)
    return frames


def _svgf_frames(case, seed):
    """Four frames of a panning camera; a plane appears in the third of them."""
    spec = scene.pan_with_disocclusion(case["w"], case["h"], seed=int(seed) % 100000)
    count = {"cut": 1, "host": 2}.get(case["kind"], 4)
    return _spec_frames(spec, 28, count, case["half"], case["kind"] != "ref")


def _batch_sizes(case):
    return [(s.width, s.height) for s in scene.stream_specs(case["n"], STREAM_SIZES, seed=3)]


def _batch_frames(case, seed):
    """Two frames of every stream: [frame][stream]."""
    specs = scene.stream_specs(case["n"], STREAM_SIZES, seed=3)
    per = []
    for k, s in enumerate(specs):
        s.seed = (int(seed) % 100000) * 97 + k
        per.append(_spec_frames(s, 1, 2, case["half"], True))
    return [[p[t] for p in per] for t in range(2)]


def _fog(case, seed):
    sc = fog_scene.FogScene(fog_scene.fog_config(seed=int(seed) % 100000, width=case["w"], height=case["h"],
                                                 depth=case["d"]), "cuda")
    dt = torch.float16 if case["half"] else torch.float32
    return [(sc.param_args(t), sc.inject(t, dt)) for t in range(1, 4)]


def _hdr(case, seed):
    spec = scene.pan_with_disocclusion(case["w"], case["h"], seed=int(seed) % 100000)
    r = scene.PlaneScene(spec, "cuda").frame(30)["radiance"]
    return r.to(torch.float16) if case["half"] else r


def _eye_sizes(case):
    sides = [8, 64, 128, 256, 32, 200, 96, 160]
    return [(sides[k % 8], sides[k % 8] if k % 3 else max(1, sides[k % 8] * 3 // 4)) for k in range(case["n"])]


def _eye_images(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    col, dep = [], []
    for w, h in _eye_sizes(case):
        c = torch.rand((h, w, 4), generator=g, device="cuda")
        col.append((c * 255).to(torch.uint8) if case["colour"] == "bgra" else c.half() if case["colour"] == "half" else c)
        dep.append(torch.rand((h, w), generator=g, device="cuda"))
    return col, dep


# ----------------------------------------------------------- prepare / run ----


def _pin(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, t=0)
    if kind in ("ref", "full", "cut", "host"):
        w, h, half = case["w"], case["h"], case["half"]
        s["den"] = tg.Denoiser(w, h, mode=tg.MODE_REF_EXACT if kind == "ref" else tg.MODE_FULL,
                               storage=tg.STORAGE_FP16 if half else tg.STORAGE_FP32)
        s["frames"] = _svgf_frames(case, seed)
        dt = torch.float16 if half else torch.float32
        if kind == "host":
            s["frames"] = [{k: _pin(v) for k, v in f.items()} for f in s["frames"]]
            s["outs"] = [torch.empty((h, w, 4), dtype=dt, pin_memory=True) for _ in range(3)]
        else:
            s["outs"] = [torch.empty((h, w, 4), dtype=dt, device="cuda") for _ in range(2)]
        if kind != "cut":
            for _ in range(WARM):
                run(s)
        if kind == "host":
            s["den"].synchronize()
    elif kind == "batch":
        sizes = _batch_sizes(case)
        s["batch"] = Batch(sizes, storage=tg.STORAGE_FP16 if case["half"] else tg.STORAGE_FP32)
        s["frames"] = _batch_frames(case, seed)
        dt = torch.float16 if case["half"] else torch.float32
        s["outs"] = [[torch.empty((h, w, 4), dtype=dt, device="cuda") for w, h in sizes] for _ in range(2)]
        s["ids"] = list(range(len(sizes)))
        for _ in range(WARM):
            run(s)
    elif kind == "fog":
        dt = torch.float16 if case["half"] else torch.float32
        s["filter"] = tg.FogFilter(case["w"], case["h"], case["d"], dtype=dt)
        s["frames"] = [(tg.fog_params(**a), v) for a, v in _fog(case, seed)]
        for _ in range(2):
            run(s)
    elif kind == "post":
        s["pp"] = tg.PostProcessor(case["w"], case["h"])
        s["hdr"] = _hdr(case, seed)
        s["order"] = "rgba" if case["out"] == "rgba" else "bgra"
        dt = torch.float32 if case["out"] == "float" else torch.uint8
        s["outs"] = [torch.empty((case["h"], case["w"], 4), dtype=dt, device="cuda") for _ in range(2)]
    else:
        # the entities' brains map the ring as shared memory: the program owns it and reads its own views of it
        sizes, up = _eye_sizes(case), lambda v: (v + 15) // 16 * 16  # noqa: E731
        room = 3 * sum(up(3 * w * h) + up(4 * w * h) for w, h in sizes)
        region = np.zeros(room + 64, np.uint8)
        skip = -region.ctypes.data % 64
        s["region"] = region[skip:skip + room]
        s["eyes"] = tg.EyeReadback(sizes, host_buffer=s["region"])
        s["images"] = _eye_images(case, seed)
        for _ in range(2):  # the ring is read two frames behind
            s["eyes"].submit(s["t"], *s["images"])
            s["t"] += 1
    return s


def _own_view(region, a):
    """The program's view of its own region where the readback's view `a` lies."""
    at = a.ctypes.data - region.ctypes.data
    return region[at:at + a.nbytes].view(a.dtype).reshape(a.shape)


def run(s):
    kind, t = s["kind"], s["t"]
    s["t"] = t + 1
    if kind == "eye":
        s["eyes"].submit(t, *s["images"])
        return [[_own_view(s["region"], a) for a in eye[:2]] for eye in s["eyes"].acquire(t - 2)]
    if kind == "fog":
        params, inject = s["frames"][t % len(s["frames"])]
        return s["filter"].step(params, inject)
    out = s["outs"][t % len(s["outs"])]
    if kind == "post":
        return s["pp"].process(s["hdr"], out, order=s["order"])
    frame = s["frames"][t % len(s["frames"])]
    if kind == "batch":
        return s["batch"].denoise(s["ids"], frame, out)
    if kind == "host":
        return s["den"].denoise_host(**frame, out=out)
    if kind == "cut":
        s["den"].reset()
    return s["den"].denoise(**frame, out=out)


# -------------------------------------------------------------------- work ----


def _svgf_work(w, h, full, half):
    """Inputs read once, state read and written once, the output written once; the operations of the taps."""
    c, m = (8, 4) if half else (16, 8)
    if not full:
        return dict(bytes=w * h * (c + 2 * m + c), flops=w * h * (3 * 25 * 13 + 20))
    inputs = 8 + 4 + 4 + 8 if half else 16 + 4 + 12 + 8
    state = 2 * (8 + 8 + 4) if half else 2 * (16 + 16 + 8)
    # a tap of a level: 5 for the normals' product, 2 + 2 for the depth and luminance stops, 4 for the two powers,
    # 10 for the sums; about 60 to set a pixel up, about 90 for the temporal pass
    return dict(bytes=w * h * (inputs + state + c), flops=w * h * (5 * (25 * 23 + 60) + 90))


def work(case):
    kind = case["kind"]
    if kind in ("ref", "full", "host"):
        return _svgf_work(case["w"], case["h"], kind != "ref", case["half"])
    if kind == "cut":
        b = _svgf_work(case["w"], case["h"], True, case["half"])
        return dict(bytes=b["bytes"], flops=b["flops"] + case["w"] * case["h"] * 49 * 18)
    if kind == "batch":
        parts = [_svgf_work(w, h, True, case["half"]) for w, h in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "fog":
        n = case["w"] * case["h"] * case["d"]
        return dict(bytes=n * 3 * (8 if case["half"] else 16), flops=n * 220)
    if kind == "post":
        n = case["w"] * case["h"]
        return dict(bytes=n * ((8 if case["half"] else 16) + (16 if case["out"] == "float" else 4)), flops=n * 160)
    n = sum(w * h for w, h in _eye_sizes(case))
    return dict(bytes=n * ({"bgra": 4, "half": 8, "float": 16}[case["colour"]] + 4 + 7), flops=n * 6)


# ------------------------------------------------------------------- exact ----

LUMA = (0.2126, 0.7152, 0.0722)


def _lum(c):
    return LUMA[0] * c[0] + LUMA[1] * c[1] + LUMA[2] * c[2]


def _planes(t):
    """(h, w, c) or (h, w) as float64 (c, h, w)."""
    t = t.cuda().double()
    return t[None] if t.dim() == 2 else t.permute(2, 0, 1).contiguous()


def _unit_normal(t):
    if t.dtype != torch.int16:
        return _planes(t)[:3]
    p = torch.clamp(_planes(t) / 32767.0, min=-1.0)
    z = 1 - p[0].abs() - p[1].abs()
    one = torch.ones_like(z)
    sx, sy = torch.where(p[0] >= 0, one, -one), torch.where(p[1] >= 0, one, -one)
    x = torch.where(z < 0, (1 - p[1].abs()) * sx, p[0])
    y = torch.where(z < 0, (1 - p[0].abs()) * sy, p[1])
    n = torch.stack([x, y, z])
    return n / n.norm(dim=0, keepdim=True)


B3 = (1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16)


def _ref_frame(rad, mom):
    """One frame of the engine's chain: moments, then three wavelet passes with clamped taps."""
    c = _planes(rad)[:3]
    h, w = c.shape[1:]
    l = _lum(c)
    mom = mom + 0.2 * (torch.stack([l, l * l]) - mom)
    alpha = (torch.clamp(mom[1] - mom[0] ** 2, min=0) + 1e-4).sqrt()
    sigma = torch.clamp(2 * alpha, min=1e-4)
    ys, xs = torch.arange(h, device=c.device), torch.arange(w, device=c.device)
    for s in (1, 2, 4):
        l = _lum(c)
        acc, ws = torch.zeros_like(c), torch.zeros_like(l)
        for dy in range(-2, 3):
            yy = (ys + s * dy).clamp(0, h - 1)
            for dx in range(-2, 3):
                xx = (xs + s * dx).clamp(0, w - 1)
                q = c[:, yy][:, :, xx]
                wt = B3[dx + 2] * B3[dy + 2] * torch.exp(-(_lum(q) - l).abs() / sigma)
                acc += wt * q
                ws += wt
        c = torch.where(ws > 1e-6, acc / ws, c)
    return torch.cat([c, torch.ones_like(c[:1])]), mom


def _pad(t, r):
    return torch.nn.functional.pad(t, (r, r, r, r))


def _one_sided(z, dim):
    d = z.diff(dim=dim)
    n = z.shape[dim]
    if n == 1:
        return torch.zeros_like(z)
    left, right = torch.cat([d.narrow(dim, 0, 1), d], dim), torch.cat([d, d.narrow(dim, n - 2, 1)], dim)
    return torch.where(left.abs() <= right.abs(), left, right)


def _full_frame(rad, depth, normal, motion, state):
    """One frame of the full filter (temporal pass, variance estimate, five levels); state: guide, history, moments."""
    c, z, n = _planes(rad)[:3], _planes(depth)[0], _unit_normal(normal)
    mv = _planes(motion)
    h, w = z.shape
    dev = z.device
    gx, gy = _one_sided(z, 1), _one_sided(z, 0)
    l = _lum(c)
    if state is None:
        state = dict(z=torch.zeros_like(z), n=torch.zeros_like(n), c=torch.zeros_like(c), len=torch.zeros_like(z),
                     mu=torch.zeros_like(z), var=torch.zeros_like(z))
    px = torch.arange(w, device=dev, dtype=torch.float64)[None, :] + mv[0]
    py = torch.arange(h, device=dev, dtype=torch.float64)[:, None] + mv[1]
    x0, y0 = px.floor(), py.floor()
    fx, fy = px - x0, py - y0
    tol = 0.05 * z + 4 * (gx.abs() + gy.abs()) + 0.1
    taps, sw, lmax = [], torch.zeros_like(z), torch.zeros_like(z)
    hc, hmu = torch.zeros_like(c), torch.zeros_like(z)
    for k in range(4):
        tx, ty = x0 + (k & 1), y0 + (k >> 1)
        inside = (tx >= 0) & (ty >= 0) & (tx < w) & (ty < h)
        j = (torch.where(inside, ty, torch.zeros_like(ty)) * w + torch.where(inside, tx, torch.zeros_like(tx))).long()
        take = lambda p: p.reshape(-1)[j]  # noqa: E731
        tl = take(state["len"])
        tn = torch.stack([take(state["n"][q]) for q in range(3)])
        d = (tn * n).sum(0)
        ok = inside & (tl > 0) & ((take(state["z"]) - z).abs() <= tol) & (d >= 0) & \
            (d * d >= 0.81 * (tn * tn).sum(0) * (n * n).sum(0))
        bw = (fx if k & 1 else 1 - fx) * (fy if k >> 1 else 1 - fy) * ok
        sw += bw
        hc += bw * torch.stack([take(state["c"][q]) for q in range(3)])
        hmu += bw * take(state["mu"])
        lmax = torch.maximum(lmax, torch.where(ok, tl, torch.zeros_like(tl)))
        taps.append((bw, take(state["mu"]), take(state["var"])))
    has = sw > 0
    inv = 1 / torch.where(has, sw, torch.ones_like(sw))
    hc, hmu = hc * inv, hmu * inv
    hvar = sum(b * (v + (m - hmu) ** 2) for b, m, v in taps) * inv
    ln = torch.where(has, torch.clamp(lmax + 1, max=32), torch.ones_like(lmax))
    a = torch.clamp(1 / ln, min=0.2)
    dl = l - hmu
    tc = torch.where(has, hc + a * (c - hc), c)
    mu = torch.where(has, hmu + a * dl, l)
    mvar = torch.where(has, (1 - a) * (hvar + a * dl * dl), torch.zeros_like(l))

    def stop(np_, zp, dx, dy, sigma_z=1.0):
        """Normal and depth stops towards the neighbour at (dx, dy) pixels, from padded normals and depths."""
        d = torch.clamp((np_ * n).sum(0), min=0)
        return d ** 128, (zp - z).abs() / (sigma_z * (gx * dx + gy * dy).abs() + 1e-3)

    var = mvar
    if bool((ln < 4).any()):
        pn, pz, pm, pv = _pad(n, 3), _pad(z[None], 3)[0], _pad(mu[None], 3)[0], _pad(mvar[None], 3)[0]
        s0, s1, s2 = torch.zeros_like(z), torch.zeros_like(z), torch.zeros_like(z)
        for dy in range(-3, 4):
            for dx in range(-3, 4):
                at = (slice(3 + dy, 3 + dy + h), slice(3 + dx, 3 + dx + w))
                wn, ez = stop(pn[(slice(None),) + at], pz[at], dx, dy)
                wt = wn * torch.exp(-ez)
                dm = pm[at] - mu
                s0 += wt
                s1 += wt * dm
                s2 += wt * (dm * dm + pv[at])
        est = torch.where(s0 > 0, torch.clamp(s2 / s0 - (s1 / s0) ** 2, min=0), mvar)
        var = torch.where(ln < 4, est, mvar)
    col = torch.cat([tc, var[None]])
    hist = None
    one = _pad(torch.ones_like(z)[None], 1)[0]
    for level in range(5):
        s = 1 << level
        pv = _pad(col[3:4], 1)[0]
        gv, gs = torch.zeros_like(z), torch.zeros_like(z)
        for dy in range(3):
            for dx in range(3):
                k = (2 if dy == 1 else 1) * (2 if dx == 1 else 1) / 16
                gv += k * pv[dy:dy + h, dx:dx + w]
                gs += k * one[dy:dy + h, dx:dx + w]
        sig = 4 * torch.clamp(gv / gs, min=0).sqrt() + 1e-4
        r = 2 * s
        pc, pn, pz = _pad(col, r), _pad(n, r), _pad(z[None], r)[0]
        lp = _lum(col)
        acc, ws, w2 = torch.zeros_like(tc), torch.zeros_like(z), torch.zeros_like(z)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                at = (slice(r + s * dy, r + s * dy + h), slice(r + s * dx, r + s * dx + w))
                q = pc[(slice(None),) + at]
                wn, ez = stop(pn[(slice(None),) + at], pz[at], s * dx, s * dy)
                wt = B3[dx + 2] * B3[dy + 2] * wn * torch.exp(-ez - (_lum(q) - lp).abs() / sig)
                acc += wt * q[:3]
                ws += wt
                w2 += wt * wt * q[3]
        ok = ws > 0
        inv = 1 / torch.where(ok, ws, torch.ones_like(ws))
        col = torch.where(ok, torch.cat([acc * inv, (w2 * inv * inv)[None]]), col)
        if level == 0:
            hist = col[:3].clone()
    out = torch.cat([col[:3], torch.ones_like(col[:1])])
    return out, dict(z=z, n=n, c=hist, len=ln, mu=mu, var=mvar)


def _exact_svgf(frames, passes, full):
    state = None
    if not full:
        state = torch.zeros((2,) + tuple(frames[0]["radiance"].shape[:2]), dtype=torch.float64, device="cuda")
    for t in range(passes):
        f = frames[t % len(frames)]
        out, state = _full_frame(f["radiance"], f["depth"], f["normal"], f["motion"], state) if full \
            else _ref_frame(f["radiance"], state)
    return out.permute(1, 2, 0).contiguous()


def _exact_fog(frames, passes):
    hist = torch.zeros_like(frames[0][1], dtype=torch.float64).permute(3, 0, 1, 2).contiguous()
    for t in range(passes):
        a, raw = frames[t % len(frames)]
        W, H, D, near, far = a["width"], a["height"], a["depth"], a["near_plane"], a["far_plane"]
        f32 = lambda v: torch.as_tensor(np.asarray(v, np.float64).astype(np.float32), device="cuda").double()  # noqa: E731
        ivp, pvp, cam = f32(a["inv_view_projection"]), f32(a["prev_view_projection"]), f32(a["camera_pos"])
        near, far, alpha = (float(np.float32(v)) for v in (near, far, a["alpha"]))
        q = raw.double().permute(3, 0, 1, 2).contiguous()
        pad = torch.nn.functional.pad(q, (1, 1, 1, 1))
        one = torch.nn.functional.pad(torch.ones((1, 1, H, W), dtype=torch.float64, device="cuda"), (1, 1, 1, 1))[0, 0]
        s, cnt = torch.zeros_like(q), torch.zeros((H, W), dtype=torch.float64, device="cuda")
        for dy in range(3):
            for dx in range(3):
                s += pad[:, :, dy:dy + H, dx:dx + W]
                cnt += one[dy:dy + H, dx:dx + W]
        mean = s / cnt
        if not a["history_valid"]:
            hist = mean
            continue
        ar = lambda n: torch.arange(n, device="cuda", dtype=torch.float64)  # noqa: E731
        nx = ((ar(W) + 0.5) / W * 2 - 1)[None, :].expand(H, W)
        ny = (1 - (ar(H) + 0.5) / H * 2)[:, None].expand(H, W)
        p = torch.stack([nx, ny, torch.zeros_like(nx), torch.ones_like(nx)], -1) @ ivp.T
        ray = p[..., :3] / p[..., 3:] - cam
        ray = ray / ray.norm(dim=-1, keepdim=True)
        fwd = ivp[:, 3][:3] / ivp[3, 3] - cam
        fwd = fwd / fwd.norm()
        rdf = (ray * fwd).sum(-1).clamp_min(1e-4)
        vz = near * (far / near) ** ((ar(D) + 0.5) / D)
        wpos = cam + ray[None] * (vz[:, None, None] / rdf[None])[..., None]
        pc = torch.cat([wpos, torch.ones_like(wpos[..., :1])], -1) @ pvp.T
        pw = pc[..., 3]
        ok = (pw > 1e-4) & (pw >= near) & (pw <= far)
        safe = torch.where(ok, pw, torch.ones_like(pw))
        fx = (pc[..., 0] / safe * 0.5 + 0.5) * W
        fy = (-pc[..., 1] / safe * 0.5 + 0.5) * H
        fz = torch.log(safe / near) / math.log(far / near) * D - 0.5
        ok &= (fx >= 0) & (fx < W) & (fy >= 0) & (fy < H) & (fz >= 0) & (fz < D)
        zero = torch.zeros_like(fx)
        fx, fy, fz = (torch.where(ok, v, zero) for v in (fx, fy, fz))
        flat = hist.reshape(4, -1)
        got = torch.zeros_like(mean)
        for k in range(8):
            ix, iy, iz = fx.floor() + (k & 1), fy.floor() + ((k >> 1) & 1), fz.floor() + (k >> 2)
            wt = 1.0
            for v, i, b in ((fx, ix, k & 1), (fy, iy, (k >> 1) & 1), (fz, iz, k >> 2)):
                fr = v - v.floor()
                wt = wt * (fr if b else 1 - fr)
            j = ((iz.clamp(0, D - 1) * H + iy.clamp(0, H - 1)) * W + ix.clamp(0, W - 1)).long()
            got += wt * flat[:, j]
        hist = torch.where(ok, got + (mean - got) * alpha, mean)
    return hist.permute(1, 2, 3, 0).contiguous()


def _exact_post(hdr):
    """The bloom chain and the post pass; display bytes have no exact value, so only the float image does."""
    c = _planes(hdr)[:3]
    H, W = c.shape[1:]
    dev = c.device

    def at(p, x, y):
        return p[:, y.clamp(0, p.shape[1] - 1)][:, :, x.clamp(0, p.shape[2] - 1)]

    ar = lambda n: torch.arange(n, device=dev)  # noqa: E731
    bw, bh = max(W // 2, 1), max(H // 2, 1)
    n = min(int(math.floor(math.log2(max(bw, bh)))) + 1, 6)
    pos = c.clamp(min=0)
    pos = pos * (_lum(pos) >= 1.0)
    wt = 1 / (1 + _lum(pos))
    num, den = 0, 0
    for k in range(4):
        x, y = 2 * ar(bw) + (k & 1), 2 * ar(bh) + (k >> 1)
        num = num + at(pos * wt, x, y)
        den = den + at(wt[None], x, y)
    mips = [num / den.clamp(min=1e-7)]
    for i in range(1, n):
        x, y = ar(max(bw >> i, 1)), ar(max(bh >> i, 1))
        mips.append(sum(at(mips[-1], 2 * x + (k & 1), 2 * y + (k >> 1)) for k in range(4)) / 4)
    for i in range(n - 2, -1, -1):
        x, y = ar(mips[i].shape[2]) // 2, ar(mips[i].shape[1]) // 2
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                mips[i] = mips[i] + (2 - abs(dx)) * (2 - abs(dy)) / 16 * at(mips[i + 1], x + dx, y + dy)
    lit = c + 0.095 * at(mips[0], ar(W) // 2, ar(H) // 2)
    ox = ((ar(W).double() + 0.5) / W - 0.5)[None, :].expand(H, W)
    oy = ((ar(H).double() + 0.5) / H - 0.5)[:, None].expand(H, W)
    d2 = ox * ox + oy * oy
    px, py = (ox * d2 * 0.0015 * W).trunc().long(), (oy * d2 * 0.0015 * H).trunc().long()
    gx, gy = ar(W)[None, :].expand(H, W), ar(H)[:, None].expand(H, W)
    pick = lambda ch, s: lit[ch][(gy + s * py).clamp(0, H - 1), (gx + s * px).clamp(0, W - 1)]  # noqa: E731
    v = torch.stack([pick(0, 1), lit[1], pick(2, -1)])
    m1 = torch.tensor([[0.59719, 0.35458, 0.04823], [0.07600, 0.90834, 0.01566], [0.02840, 0.13383, 0.83777]])
    m2 = torch.tensor([[1.60475, -0.53108, -0.07367], [-0.10208, 1.10813, -0.00605], [-0.00327, -0.07276, 1.07602]])
    v = torch.einsum("ij,jhw->ihw", m1.double().to(dev), v)
    v = (v * (v + 0.0245786) - 0.000090537) / (v * (0.983729 * v + 0.4329510) + 0.238081)
    v = torch.einsum("ij,jhw->ihw", m2.double().to(dev), v).clamp(0, 1)
    v = torch.where(v <= 0.0031308, 12.92 * v, 1.055 * v.clamp(min=1e-12) ** (1 / 2.4) - 0.055)
    l = _lum(v)
    cool = torch.stack([0.9 * l, 0.95 * l, 1.1 * l])
    v = (v + 0.15 * (cool - v)) * (1 - 1.5 * d2).clamp(0, 1)
    return torch.cat([v, torch.ones_like(v[:1])]).permute(1, 2, 0).contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ref", "full", "cut", "host"):
        return _exact_svgf(_svgf_frames(case, seed), 1 if kind == "cut" else WARM + 1, kind != "ref")
    if kind == "batch":
        frames = _batch_frames(case, seed)
        return [_exact_svgf([f[k] for f in frames], WARM + 1, True) for k in range(case["n"])]
    if kind == "fog":
        return _exact_fog(_fog(case, seed), 3)
    if kind == "post" and case["out"] == "float":
        return _exact_post(_hdr(case, seed))
    return None
