"""What this framework's users have it do, as cases a benchmark can run: frames of every size rendered through resident
scenes, moving crowds, both denoisers, the denoiser's training, a moving sun and a burst of served requests.

`listed()` names the cases, `draw(rng)` makes another of the same ranges, `prepare(case, seed)` is what a program holds
before the call, `run(state)` one pass through the public entry points, `work(case)` what a pass cannot do without, and
`exact(case, seed)` the pass's result in 64 bits where plain torch can give it.

A case's seed moves the camera along the scene's path (or the walkers, or the sun), and seeds the sampler, the
network's weights and its training data; the geometry of a named scene is the same for every seed, as a resident
scene's is, and is generated once a process.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from threert_b200 import Gpu, crowd, prep, scenes, serve, unet
from threert_b200 import _native as N

PIXEL = 80          # bytes of a Pixel record
FPS = crowd.FPS


def listed():
    return [
        # The smallest call: a thumbnail of a small scene, its accum read back (a preview, a tool's icon, a test).
        {"name": "thumbnail", "path": "render", "scene": "cornell", "w": 64, "h": 64, "spp": 1, "bounces": 5,
         "back": True},
        # The Cornell box at its benchmark size: few triangles, deep paths, read back.
        {"name": "cornell", "path": "render", "scene": "cornell", "w": 256, "h": 256, "spp": 16, "bounces": 5,
         "back": True},
        # The noisy half of a denoiser's training pair: a small city, a small square view, the depth guide on.
        {"name": "pair_view", "path": "render", "scene": "town", "w": 128, "h": 128, "spp": 4, "bounces": 4,
         "depth": True, "back": True},
        # A frame of the city fly-through (the headline workload), its accum handed to a consumer on the device.
        {"name": "city_frame", "path": "render", "scene": "city", "w": 1280, "h": 720, "spp": 1, "bounces": 4},
        # A still of the city: the largest image, several samples (many waves a call).
        {"name": "city_still", "path": "render", "scene": "city", "w": 1920, "h": 1080, "spp": 16, "bounces": 4},
        # A frame of the walking crowd, one pose shared by 5,000 walkers: records and palette in, deformation, top
        # tree, render.
        {"name": "crowd_frame", "path": "crowd", "walkers": 5000, "groups": 1, "w": 1280, "h": 720, "spp": 1,
         "bounces": 3},
        # The same with many poses (5 M skinned triangles): the deformation carries the frame.
        {"name": "crowd_poses", "path": "crowd", "walkers": 2000, "groups": 256, "w": 640, "h": 360, "spp": 1,
         "bounces": 3},
        # The learned denoiser on a rendered 720p frame, the image read back.
        {"name": "denoise_net", "path": "denoise", "w": 1280, "h": 720, "spp": 4},
        # The fallback denoiser on the same.
        {"name": "denoise_atrous", "path": "atrous", "w": 1280, "h": 720, "spp": 4, "iterations": 4},
        # A step of the denoiser's training: 16 crops of 64 x 64, forward, backward, Adam; its gradients read back.
        {"name": "train_step", "path": "train", "batch": 16, "h": 64, "w": 64},
        # The sun moved: the sky baked again into the resident scene, and a preview frame under it.
        {"name": "moving_sun", "path": "sun", "sky_w": 1024, "sky_h": 512, "w": 256, "h": 144, "spp": 1, "bounces": 4},
        # A burst of requests of mixed sizes and sample counts to the server, on resident scenes.
        {"name": "serve_burst", "path": "serve", "requests": 12, "side": 256, "spp": 16, "bounces": 4},
    ]


def _span(rng, lo, hi):
    """An integer from lo to hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["render", "render", "render", "render", "crowd", "denoise", "atrous", "train", "sun", "serve"])
    if path == "render":
        scene = rng.choice(["cornell", "town", "city"])
        w = _span(rng, 32, 1920)
        h = max(16, min(1080, int(w * rng.uniform(0.5, 1.0))))
        most = max(1, min(64, 16 * 1920 * 1080 // (w * h) // 2))
        return {"path": "render", "scene": scene, "w": w, "h": h, "spp": _span(rng, 1, most),
                "bounces": rng.randint(2, 8 if scene == "cornell" else 5), "depth": rng.random() < 0.3,
                "back": rng.random() < 0.4}
    if path == "crowd":
        groups = _span(rng, 1, 256)
        return {"path": "crowd", "walkers": max(groups, _span(rng, 300, 5000)), "groups": groups,
                "w": _span(rng, 200, 1280), "h": _span(rng, 120, 720), "spp": 1, "bounces": 3}
    if path in ("denoise", "atrous"):
        w, h = _span(rng, 16, 160) * 8, _span(rng, 10, 90) * 8
        if path == "denoise":
            return {"path": "denoise", "w": w, "h": h, "spp": rng.choice([1, 2, 4])}
        return {"path": "atrous", "w": w + rng.randint(0, 7), "h": h + rng.randint(0, 7), "spp": rng.choice([1, 2, 4]),
                "iterations": rng.choice([3, 4, 5])}
    if path == "train":
        return {"path": "train", "batch": _span(rng, 1, 32), "h": rng.choice([32, 64, 72, 96, 128]),
                "w": rng.choice([32, 40, 64, 96, 128])}
    if path == "sun":
        w = rng.choice([128, 256, 512, 1024])
        return {"path": "sun", "sky_w": w, "sky_h": w // 2, "w": _span(rng, 64, 512), "h": _span(rng, 36, 288),
                "spp": rng.choice([1, 2, 4]), "bounces": 4}
    return {"path": "serve", "requests": rng.randint(2, 16), "side": _span(rng, 64, 512), "spp": _span(rng, 1, 16),
            "bounces": 4}


# ---- what a program holds before the call ----------------------------------------------------------------------------

_made = {}


def _once(key, make):
    if key not in _made:
        _made[key] = make()
    return _made[key]


def _gpu() -> Gpu:
    return _once("gpu", lambda: Gpu(0))


def _prepared(scene):
    """The named scene's buffers (its atmosphere baked)."""
    def make():
        if scene == "cornell":
            d = scenes.cornell()
        elif scene == "town":
            d = scenes.city(n_objects=300, width=128, height=128, seed=5, extent=100.0, n_emitters=60, box_segments=2,
                            sphere_slices=12, sphere_stacks=10, sky_size=(256, 128))
        else:
            d = scenes.city()
        P = prep.prepare(d)
        _gpu().upload(P).close()  # (bakes the sky into the prepared buffers)
        return P
    return _once(scene, make)


def _view(scene, P, rng, w, h, bounces):
    """Params of one view: the camera somewhere on the scene's path, a sampler seed of its own."""
    p = prep.params_with(P.params, max_bounces=bounces, seed=int(rng.integers(1, 1 << 30)))
    p[16], p[17] = w, h
    p[7] = np.float32(w / h).view(np.uint32)
    if scene == "cornell":
        at = (float(rng.uniform(-0.4, 0.4)), float(rng.uniform(0.7, 1.3)), float(rng.uniform(3.5, 4.0)))
        return prep.set_camera(p, prep.Camera.look_at(at, (0.0, 1.0, 0.0), 39.0, w, h))
    seed, extent = (5, 100.0) if scene == "town" else (1, 500.0)
    return prep.set_camera(p, scenes.city_camera(int(rng.integers(0, 240)), 240, seed, w, h, extent))


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def _crowd(case):
    def make():
        c = crowd.crowd(n=case["walkers"], groups=case["groups"], max_depth=case["bounces"])
        P = prep.prepare(c.desc)
        _gpu().upload(P).close()
        return c, P, crowd.deform_jobs(P, c)
    return _once(("crowd", case["walkers"], case["groups"], case["bounces"]), make)


def _sun(atm, elevation, azimuth):
    atm.sun_dir = (N.f32 * 3)(math.cos(elevation) * math.cos(azimuth), math.sin(elevation),
                              math.cos(elevation) * math.sin(azimuth))
    return atm


def _noisy(case, seed):
    """A scene just rendered with the depth guide: what both denoisers start from."""
    rng = np.random.default_rng(seed)
    P = _prepared("town")
    S = _gpu().upload(P)
    params = _view("town", P, rng, case["w"], case["h"], 4)
    S.render_raw(params, case["spp"], flags=N.TRT_RENDER_DEPTH, read=False, stats=False)
    return S


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    path = case["path"]
    st = {"path": path}
    if path == "render":
        P = _prepared(case["scene"])
        st["S"] = _gpu().upload(P)
        st["params"] = _view(case["scene"], P, rng, case["w"], case["h"], case["bounces"])
        st["spp"] = case["spp"]
        st["flags"] = N.TRT_RENDER_DEPTH if case.get("depth") else 0
        shape = (case["w"] * case["h"], N.PIXEL_FLOATS)
        st["host"] = _pinned(shape) if case.get("back") else None
        st["out"] = None if case.get("back") else torch.empty(shape, dtype=torch.float32, device="cuda")
    elif path == "crowd":
        c, P, (corners, jobs) = _crowd(case)
        st["S"] = _gpu().upload(P)
        st["S"].deform_setup(corners, jobs)
        frame = int(rng.integers(0, 600))
        t = frame / FPS
        st["at"] = crowd.records(P)[0] * 16
        st["records"] = crowd.frame_records(P, c, t)
        st["palette"] = crowd.palettes(t, c.phase, c.scale)
        p = prep.params_with(P.params, seed=int(rng.integers(1, 1 << 30)))
        p[16], p[17] = case["w"], case["h"]
        p[7] = np.float32(case["w"] / case["h"]).view(np.uint32)
        st["params"] = prep.set_camera(p, crowd.crowd_camera(frame, case["w"], case["h"], c.extent))
        st["spp"] = case["spp"]
        st["out"] = torch.empty((case["w"] * case["h"], N.PIXEL_FLOATS), dtype=torch.float32, device="cuda")
    elif path == "denoise":
        st["net"] = unet.UNet(0, max_batch=1, max_h=case["h"], max_w=case["w"])
        st["net"].set_params(unet.init_params(seed))
        st["S"] = _noisy(case, seed)
    elif path == "atrous":
        st["S"] = _noisy(case, seed)
        st["iterations"] = case["iterations"]
    elif path == "train":
        st["net"] = unet.UNet(0, max_batch=case["batch"], max_h=case["h"], max_w=case["w"])
        st["net"].set_params(unet.init_params(seed))
        st["x"], st["t"] = _crops(case, seed)
    elif path == "sun":
        P = _prepared_sky(case)
        st["S"] = _gpu().upload(P)
        atm, st["sun_light"] = _made[("sky", case["sky_w"])][1]
        st["atm"] = _sun(N.Atmosphere.from_buffer_copy(atm), math.radians(float(rng.uniform(5.0, 60.0))),
                         math.radians(float(rng.uniform(0.0, 360.0))))
        st["floor"] = P.info["env_nee_floor"]
        st["params"] = _view("town", P, rng, case["w"], case["h"], case["bounces"])
        st["spp"] = case["spp"]
        st["out"] = torch.empty((case["w"] * case["h"], N.PIXEL_FLOATS), dtype=torch.float32, device="cuda")
    else:
        names = ("cornell", "town")
        st["server"] = serve.Server(_gpu())
        st["scenes"] = [_gpu().upload(_prepared(n)) for n in names]
        st["asks"] = []
        for k in range(case["requests"]):
            side = case["side"] << (k % 2)           # two sizes, two sample counts, two scenes
            spp = case["spp"] if k % 3 else 1
            p = _view(names[k % 2], _prepared(names[k % 2]), rng, side, side, case["bounces"])
            st["asks"].append((k % 2, p, spp))
        st["held"] = []
    return st


def _prepared_sky(case):
    def make():
        P = prep.prepare(scenes.city(n_objects=300, width=128, height=128, seed=5, extent=100.0, n_emitters=60,
                                     box_segments=2, sphere_slices=12, sphere_stacks=10,
                                     sky_size=(case["sky_w"], case["sky_h"])))
        pending = P.sky_pending
        _gpu().upload(P).close()
        return P, pending
    return _once(("sky", case["sky_w"]), make)[0]


def _crops(case, seed):
    """Feature and target crops with the ranges a rendered pair has: log radiance, albedo, unit normals, log depth and
    log variance, piecewise smooth with noise on the radiance."""
    rng = np.random.default_rng(seed)
    b, h, w = case["batch"], case["h"], case["w"]
    low = rng.random((b, h // 8, w // 8, 8)).astype(np.float32)
    base = low.repeat(8, 1).repeat(8, 2)
    clean = np.log1p(3.0 * base[..., 0:3] ** 2)
    noise = rng.standard_normal((b, h, w, 3)).astype(np.float32)
    n = base[..., 3:6] * 2.0 - 1.0
    n = n / np.maximum(np.linalg.norm(n, axis=-1, keepdims=True), 1e-3)
    x = np.concatenate([np.maximum(clean + 0.3 * noise, 0.0), base[..., 0:3], n, np.log1p(2.0 * base[..., 6:7]),
                        np.log1p(base[..., 7:8])], -1)
    return np.ascontiguousarray(x, np.float32), np.ascontiguousarray(clean, np.float32)


# ---- one pass --------------------------------------------------------------------------------------------------------


def run(st):
    path = st["path"]
    if path == "render":
        S = st["S"]
        if st["host"] is not None:
            acc, _ = S.render_raw(st["params"], st["spp"], flags=st["flags"], out=st["host"].numpy())
            return acc
        S.render_raw(st["params"], st["spp"], flags=st["flags"], read=False, stats=False)
        S.accum_copy(st["out"].data_ptr(), st["out"].nbytes)
        return st["out"]
    if path == "crowd":
        S = st["S"]
        S.update(3, st["at"], st["records"])
        S.deform(st["params"], st["palette"], stats=False)
        S.render_raw(st["params"], st["spp"], read=False, stats=False)
        S.accum_copy(st["out"].data_ptr(), st["out"].nbytes)
        return st["out"]
    if path == "denoise":
        return st["net"].denoise(st["S"])[0]
    if path == "atrous":
        return st["S"].denoise_atrous(st["iterations"])[0]
    if path == "train":
        loss, grads, _ = st["net"].step(st["x"], st["t"], lr=1e-3, grads=True)
        return {"loss": loss, "grads": grads}
    if path == "sun":
        p = st["params"].copy()
        S = st["S"]
        r = S.set_sky(st["atm"], st["sun_light"], st["floor"], p)
        S.render_raw(p, st["spp"], read=False, stats=False)
        S.accum_copy(st["out"].data_ptr(), st["out"].nbytes)
        return {"accum": st["out"], "sun": np.array(r.sun_illuminance, np.float32)}
    srv = st["server"]
    for r in st["held"]:
        srv.release(r)
    asks = [serve.Request(k, p, spp) for k, p, spp in st["asks"]]
    for r in asks:
        srv.submit(st["scenes"][r.scene], r)
    done = 0
    while done < len(asks):
        done += len(srv.poll(wait_ms=100))
    st["held"] = asks
    return [r.accum for r in asks]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

TRIS = {"cornell": 36, "town": 45_000, "city": 1_984_402}


def _render_work(paths, pixels, bounces, tris):
    """Paths of up to `bounces` + 1 vertices (half of them lost on the way), a closest and two shadow rays a vertex; a
    ray has to pass about log2(tris) levels of boxes (two of 13 operations each) and a couple of triangles (50 each), a
    vertex to be shaded (about 500). The accum is written once; each triangle's record and tree read at most once."""
    vertices = paths * (1 + bounces) * 0.5
    ray = math.log2(max(2, tris)) * 26 + 100
    return {"bytes": PIXEL * pixels + min(tris * 80, vertices * 3 * 80), "flops": vertices * (3 * ray + 500)}


def _net_macs(pixels):
    levels = [pixels, pixels / 4, pixels / 16, pixels / 64]
    at = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
    return sum(9 * cin * cout * levels[l] for (cin, cout), l in zip(unet.LAYERS, at))


def work(case):
    path = case["path"]
    if path == "render":
        px = case["w"] * case["h"]
        return _render_work(px * case["spp"], px, case["bounces"], TRIS[case["scene"]])
    if path == "crowd":
        px = case["w"] * case["h"]
        w = _render_work(px * case["spp"], px, case["bounces"], 20_160)
        # every posed triangle's record and box written, its vertices posed (half a vertex a triangle)
        tris = 20_160 * case["groups"]
        w["bytes"] += tris * (48 + 32 + 48)
        w["flops"] += tris * 150 + case["walkers"] * 20 * 40
        return w
    if path == "denoise":
        px = case["w"] * case["h"]
        return {"bytes": px * (PIXEL + 12) + 4 * unet.param_count(), "flops": 2 * _net_macs(px)}
    if path == "atrous":
        px = case["w"] * case["h"]
        return {"bytes": px * (PIXEL + 12), "flops": px * case["iterations"] * 25 * 50}
    if path == "train":
        px = case["batch"] * case["h"] * case["w"]
        return {"bytes": px * 14 * 4 + 9 * 4 * unet.param_count(), "flops": 6 * _net_macs(px)}
    if path == "sun":
        px, sky = case["w"] * case["h"], case["sky_w"] * case["sky_h"]
        w = _render_work(px * case["spp"], px, case["bounces"], TRIS["town"])
        w["bytes"] += sky * 12
        w["flops"] += sky / 2 * 17 * 150
        return w
    total = {"bytes": 0.0, "flops": 0.0}
    for k in range(case["requests"]):
        px = (case["side"] << (k % 2)) ** 2
        w = _render_work(px * (case["spp"] if k % 3 else 1), px, case["bounces"], TRIS[("cornell", "town")[k % 2]])
        total = {m: total[m] + w[m] for m in total}
    return total


# ---- in 64 bits ------------------------------------------------------------------------------------------------------


def exact(case, seed):
    """The denoisers and the training step; a path-traced image has no closed value (its noise is the sampler's)."""
    path = case["path"]
    if path == "atrous":
        return _exact_atrous(_accum_of(case, seed), case["w"], case["h"], case["iterations"])
    if path == "denoise":
        return _exact_denoise(_accum_of(case, seed), case["w"], case["h"], unet.init_params(seed))
    if path == "train":
        x, t = _crops(case, seed)
        return _exact_train(x, t, unet.init_params(seed))
    return None


def _accum_of(case, seed):
    S = _noisy(case, seed)
    a = torch.empty((case["h"], case["w"], N.PIXEL_FLOATS), dtype=torch.float32, device="cuda")
    S.accum_copy(a.data_ptr(), a.nbytes)
    S.close()
    a = a.double()
    return torch.where(torch.isfinite(a), a, torch.zeros_like(a))


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _mean_variance(a, cnt):
    mean = a[..., 7] / cnt
    return torch.clamp(a[..., 11] / cnt - mean * mean, min=0.0) / cnt


def _shifted(v, dy, dx, fill=0.0):
    """v[y + dy, x + dx], `fill` outside."""
    h, w = v.shape[:2]
    out = torch.full_like(v, fill)
    y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
    if y0 < y1 and x0 < x1:
        out[y0:y1, x0:x1] = v[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _exact_atrous(a, w, h, iterations):
    cnt = torch.clamp(a[..., 3], min=1.0)
    color, alb, nrm = (a[..., k:k + 3] / cnt[..., None] for k in (0, 4, 8))
    n = nrm.norm(dim=-1, keepdim=True)
    nrm = torch.where(n > 0, nrm / torch.clamp(n, min=1e-300), torch.zeros_like(nrm))
    ae = torch.clamp(alb, min=1e-3)
    cur = color / ae
    var = _mean_variance(a, cnt) / _lum(ae) ** 2
    one = torch.ones((h, w), dtype=torch.float64, device=a.device)
    for it in range(iterations):
        s, ws = torch.zeros_like(var), torch.zeros_like(var)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = (0.5 if dx == 0 else 0.25) * (0.5 if dy == 0 else 0.25)
                s += k * _shifted(var, dy, dx)
                ws += k * _shifted(one, dy, dx)
        sigma = 4.0 * torch.sqrt(torch.clamp(s / ws, min=0.0)) + 1e-4
        lp = _lum(cur)
        tot, wsum, vsum = torch.zeros_like(cur), torch.zeros_like(var), torch.zeros_like(var)
        taps = [0.375, 0.25, 0.0625]
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                o = (dy << it, dx << it)
                cq, nq, aq = _shifted(cur, *o), _shifted(nrm, *o), _shifted(alb, *o)
                wl = torch.exp(-(lp - _lum(cq)).abs() / sigma)
                wn = torch.clamp((nrm * nq).sum(-1), min=0.0) ** 64
                wa = torch.exp(-((alb - aq) ** 2).sum(-1) / 0.01)
                wt = taps[abs(dx)] * taps[abs(dy)] * wl * wn * wa * _shifted(one, *o)
                tot += cq * wt[..., None]
                vsum += wt * wt * _shifted(var, *o)
                wsum += wt
        ok = wsum > 0
        safe = torch.where(ok, wsum, torch.ones_like(wsum))
        cur = torch.where(ok[..., None], tot / safe[..., None], cur)
        var = torch.where(ok, vsum / (safe * safe), var)
    return cur * ae


def _layers(params, device):
    """The network's (weights (9, cin, cout), bias (cout,)) in 64 bits, from the flat parameters."""
    p = torch.as_tensor(params, dtype=torch.float64, device=device)
    out, o = [], 0
    for cin, cout in unet.LAYERS:
        cp = unet.r64(cout)
        wt = p[o:o + 9 * cin * cp].view(9, cin, cp)[:, :, :cout]
        out.append((wt, p[o + 9 * cin * cp:o + 9 * cin * cp + cp][:cout]))
        o += 9 * cin * cp + cp
    return out


def _conv(x, layer, relu=True):
    """A 3 x 3 convolution of x (b, h, w, cin) as nine matrix products."""
    wt, bias = layer
    b, h, w, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = bias
    for t in range(9):
        y = y + xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w] @ wt[t]
    return torch.relu(y) if relu else y


def _pool(x):
    b, h, w, c = x.shape
    return x.view(b, h // 2, 2, w // 2, 2, c).mean((2, 4))


def _up(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2)


def _network(x, layers):
    x = torch.nn.functional.pad(x, (0, 32 - x.shape[-1]))
    it = iter(layers)
    skips = []
    for _ in range(3):
        x = _conv(_conv(x, next(it)), next(it))
        skips.append(x)
        x = _pool(x)
    x = _conv(_conv(x, next(it)), next(it))
    for _ in range(3):
        x = torch.cat([_up(x), skips.pop()], -1)
        x = _conv(_conv(x, next(it)), next(it))
    return _conv(x, next(it), relu=False)


def _exact_denoise(a, w, h, params):
    cnt = torch.clamp(a[..., 3], min=1.0)
    rad, alb, nrm = (a[..., k:k + 3] / cnt[..., None] for k in (0, 4, 8))
    depth = a[..., 12] / cnt
    s = 1.0 / max(float(_lum(rad).mean()), 1e-6)
    hit = depth > 0
    sd = 1.0 / max(float(depth[hit].sum()) / max(int(hit.sum()), 1), 1e-6)
    var = _mean_variance(a, cnt)
    f = torch.cat([torch.log1p(torch.clamp(rad * s, min=0.0)), alb, nrm,
                   torch.log1p(torch.clamp(depth * sd, min=0.0))[..., None],
                   torch.log1p(torch.clamp(var * s * s, min=0.0))[..., None]], -1)
    with torch.no_grad():
        y = _network(f[None], _layers(params, a.device))[0]
    return torch.clamp(torch.expm1(y), min=0.0) / s


def _exact_train(x, t, params):
    dev = torch.device("cuda")
    p = torch.as_tensor(params, dtype=torch.float64, device=dev).requires_grad_(True)
    y = _network(torch.as_tensor(x, dtype=torch.float64, device=dev), _layers(p, dev))
    loss = (y - torch.as_tensor(t, dtype=torch.float64, device=dev)).abs().mean()
    loss.backward()
    return {"loss": float(loss), "grads": p.grad}
