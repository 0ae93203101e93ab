"""Performance cases: the calls that a user of this renderer makes, through the public
Python entry points (ctypes over the C ABI), over the range of sizes they are made at.

Each case names a kind and its sizes:
  host_rays  GpuBVHAccel.intersect / intersect_any on host arrays: the accelerator plugin's
             path, from single rays to a tile's worth
  rays       GpuBVHAccel.intersect_device on device buffers: ray batches, half coherent
             camera rays, half incoherent
  build      GpuBVHAccel.construct: the tree of a new scene, then one small ray batch
  render     GpuPathIntegrator / GpuDirectLightingIntegrator on one scene; host = 1 takes the
             host film entry point that the integrator plugin calls
  batch      GpuBatch.run: many small renders in one launch
  guided     GpuGuide.render with the learned proposal
  train      GpuGuide.train: Adam steps on collected training samples
  film       film_resolve: what every render ends in (RGBE, gamma bytes, tone mapping)
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import spica_gb300 as sg
from spica_gb300 import gpu, scenes

DEV = "cuda"
FORMATS = {"rgbe": (gpu.FILM_RGBE, 0.0), "gamma": (gpu.FILM_GAMMA_BYTES, 2.2), "reinhard": (gpu.FILM_REINHARD, 0.18),
           "drago": (gpu.FILM_DRAGO, 0.85), "durand": (gpu.FILM_DURAND, 5.0)}


def listed():
    return [
        # a few rays from one shading point or packet, as a host integrator asks for them
        {"name": "host_rays_64", "kind": "host_rays", "levels": 6, "rays": 64, "any": False},
        # the intersection workload: 1,048,576 triangles, 8M coherent and 8M incoherent rays
        {"name": "rays_closest_16m", "kind": "rays", "levels": 9, "rays": 1 << 24, "any": False},
        # an ordinary batch of occlusion tests, an odd number of them
        {"name": "rays_any_300k", "kind": "rays", "levels": 7, "rays": 300001, "any": True},
        # a new scene's tree: the 2M-triangle mid-scale scene
        {"name": "build_2m", "kind": "build", "scene": "mid", "size": 500},
        # the smallest render: a preview of the box room into a host film
        {"name": "render_box_64", "kind": "render", "scene": "box", "width": 64, "height": 64, "spp": 16, "depth": 8,
         "integrator": "path", "host": True},
        # an ordinary render at an odd size: rough dielectric and plastic among Lambert walls
        {"name": "render_material_333x217", "kind": "render", "scene": "material", "width": 333, "height": 217,
         "spp": 24, "depth": 8, "integrator": "path", "host": False},
        # the benchmark frame: 2M triangles, all three BSDF classes, area lights and sky
        {"name": "render_mid_1080p", "kind": "render", "scene": "mid", "width": 1920, "height": 1080, "spp": 16,
         "depth": 16, "integrator": "path", "host": False},
        # sixteen seeded box-room variants of 64^2 to 512^2 pixels in one launch
        {"name": "batch_16", "kind": "batch", "renders": 16, "variants": 0},
        # a guided pass of the indirect-lit room
        {"name": "guided_640x360", "kind": "guided", "width": 640, "height": 360, "spp": 8, "depth": 12},
        # Adam steps on what the last collection pass found.  The ring's order differs from run to
        # run, and so do the batches: more steps would drift too far apart to be compared
        {"name": "train_16", "kind": "train", "steps": 16, "batch": 16384},
        # a full-HD film to the bytes of a PNG
        {"name": "film_gamma_1080p", "kind": "film", "format": "gamma", "width": 1920, "height": 1080},
        # the local tone mapping operator on a 720p film
        {"name": "film_durand_720p", "kind": "film", "format": "durand", "width": 1280, "height": 720},
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["host_rays", "rays", "rays", "build", "render", "render", "render", "batch", "guided", "train",
                       "film", "film"])
    if kind == "host_rays":
        return {"kind": kind, "levels": rng.randint(3, 8), "rays": _log(rng, 1, 65536), "any": rng.random() < 0.5}
    if kind == "rays":
        return {"kind": kind, "levels": rng.randint(3, 9), "rays": _log(rng, 1000, 1 << 24), "any": rng.random() < 0.5}
    if kind == "build":
        if rng.random() < 0.5:
            return {"kind": kind, "scene": "mid", "size": rng.randint(5, 500)}
        return {"kind": kind, "scene": "sphere", "size": rng.randint(2, 9)}
    if kind == "render":
        w, h = _log(rng, 33, 1920), _log(rng, 33, 1080)
        return {"kind": kind, "scene": rng.choice(["box", "material", "conductor", "guiding", "mid", "mid"]),
                "width": w, "height": h, "spp": _log(rng, 1, max(1, min(64, 33_000_000 // (w * h)))),
                "depth": rng.randint(1, 16), "integrator": rng.choice(["path", "path", "path", "direct"]),
                "host": rng.random() < 0.4}
    if kind == "batch":
        return {"kind": kind, "renders": _log(rng, 1, 16), "variants": rng.randint(1, 9)}
    if kind == "guided":
        w = _log(rng, 64, 1280)
        return {"kind": kind, "width": w, "height": max(16, w * 9 // 16), "spp": rng.randint(1, 8),
                "depth": rng.randint(2, 12)}
    if kind == "train":
        return {"kind": kind, "steps": _log(rng, 1, 16), "batch": _log(rng, 4096, 65536)}
    return {"kind": "film", "format": rng.choice(sorted(FORMATS)), "width": _log(rng, 16, 1920),
            "height": _log(rng, 16, 1080)}


# ------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=8)
def _sphere(levels):
    return scenes.displaced_sphere(levels=levels, seed=0)


@functools.lru_cache(maxsize=8)
def _scene(name, size):
    if name == "sphere":
        return _sphere(size)
    if name == "mid":
        return scenes.mid_scale(n_instances=size)
    make = {"box": scenes.box_room, "material": scenes.material_room, "conductor": scenes.conductor_room,
            "guiding": scenes.guiding_room}
    return make[name](width=64, height=64)


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _stretched(sc, seed):
    """The scene's triangles under a seeded stretch: another mesh of the same kind."""
    rng = np.random.default_rng(seed)
    out = scenes.Scene(**{k: getattr(sc, k) for k in ("verts", "tri_mat", "materials", "tri_emit", "env")})
    s = (1.0 + 0.2 * rng.random(3)).astype(np.float32)
    out.verts = np.ascontiguousarray((sc.verts.reshape(-1, 3) * s).reshape(-1, 9))
    return out


def _rays(case, seed, sc):
    """(n, 4) origins + tmin and directions + tmax on the GPU: the first half a camera's
    raster looking at the scene from a seeded place, the second half uniform origins in its
    box and uniform directions."""
    n = case["rays"]
    v = sc.verts.reshape(-1, 3)
    lo, hi = v.min(0), v.max(0)
    g = _generator(seed)
    r = 0.5 * float(np.max(hi - lo))
    nc = n // 2
    eye = torch.randn(3, device=DEV, generator=g)
    eye = eye / eye.norm() * 3.2 * r
    fwd = -eye / eye.norm()
    side = torch.linalg.cross(fwd, torch.tensor([0.3, 0.9, 0.2], device=DEV))
    side = side / side.norm()
    up = torch.linalg.cross(side, fwd)
    w = max(1, int(math.sqrt(2 * nc)))
    h = max(1, -(-nc // w))
    i = torch.arange(nc, device=DEV)
    th = math.tan(math.radians(20.0))
    sx = (2.0 * ((i % w).float() + 0.5) / w - 1.0) * th * w / h
    sy = (1.0 - 2.0 * ((i // w).float() + 0.5) / h) * th
    org = torch.empty((n, 4), device=DEV)
    dirs = torch.empty((n, 4), device=DEV)
    org[:nc, :3] = eye
    dirs[:nc, :3] = fwd + sx[:, None] * side + sy[:, None] * up
    lo_t, ext = torch.from_numpy(lo).to(DEV), torch.from_numpy(hi - lo).to(DEV)
    org[nc:, :3] = lo_t + ext * torch.rand((n - nc, 3), device=DEV, generator=g)
    dirs[nc:, :3] = torch.randn((n - nc, 3), device=DEV, generator=g)
    d = dirs[:, :3]
    d /= d.norm(dim=1, keepdim=True)
    org[:, 3] = 0.0
    dirs[:, 3] = 1.0e32
    if case["any"]:
        dirs[:nc, 3] = 5.2 * r
        dirs[nc:, 3] = 2.0 * r * torch.rand(n - nc, device=DEV, generator=g)
    return org, dirs


def _film(case, seed):
    """A film as a 16-sample render leaves it: smooth radiance under noise, a light of
    constant radiance, black pixels."""
    W, H = case["width"], case["height"]
    g = _generator(seed)
    coarse = torch.randn((1, 3, 9, 9), device=DEV, generator=g)
    smooth = torch.nn.functional.interpolate(coarse, size=(H, W), mode="bilinear", align_corners=True)[0]
    noise = 0.3 * torch.randn((3, H, W), device=DEV, generator=g)
    rgb = 16.0 * torch.exp(smooth + noise - 1.0).permute(1, 2, 0)
    dark = torch.rand((H, W), device=DEV, generator=g) < 0.005
    rgb = torch.where(dark[..., None], torch.zeros_like(rgb), rgb)
    rgb[: max(1, H // 10), W // 3: W // 3 + max(1, W // 8)] = torch.tensor([272.0, 192.0, 64.0], device=DEV)
    film = torch.empty((H, W, 4), device=DEV)
    film[..., :3] = rgb
    film[..., 3] = 16.0
    return film


def _tree(sc):
    return sg.GpuBVHAccel(sc).construct()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("host_rays", "rays"):
        sc = _sphere(case["levels"])
        acc = _tree(sc)
        org, dirs = _rays(case, seed, sc)
        if kind == "host_rays":
            o, d = org.cpu().numpy(), dirs.cpu().numpy()
            return {"case": case, "acc": acc, "org": o[:, :3].copy(), "dir": d[:, :3].copy(), "tmax": d[:, 3].copy()}
        n = case["rays"]
        out = torch.empty(n, dtype=torch.int32, device=DEV) if case["any"] else torch.empty((n, 4), device=DEV)
        return {"case": case, "acc": acc, "org": org, "dir": dirs, "out": out}
    if kind == "build":
        sc = _stretched(_scene(case["scene"], case["size"]), seed)
        org, dirs = _rays({"rays": 4096, "any": False}, seed, sc)
        return {"case": case, "acc": sg.GpuBVHAccel(sc), "org": org, "dir": dirs,
                "out": torch.empty((4096, 4), device=DEV)}
    if kind == "render":
        sc = _scene(case["scene"], 500)
        make = sg.GpuPathIntegrator if case["integrator"] == "path" else gpu.GpuDirectLightingIntegrator
        film = None if case["host"] else torch.empty((case["height"], case["width"], 4), device=DEV)
        return {"case": case, "acc": _tree(sc), "camera": sc.camera, "integ": make(seed=seed), "film": film,
                "params": {"width": case["width"], "height": case["height"], "sampleCount": case["spp"],
                           "maxDepth": case["depth"]}}
    if kind == "batch":
        b = sg.GpuBatch(scenes.batch_variants(case["renders"], seed=case["variants"]), seed=seed, autotune=False)
        return {"case": case, "batch": b, "films": torch.empty((b.pixels, 4), device=DEV)}
    if kind == "guided":
        sc = _scene("guiding", 0)
        g = gpu.GpuGuide(_tree(sc), seed=seed)
        g.set_params(1.5 * g.params())   # lobes as peaked as some training leaves them
        film = torch.empty((case["height"], case["width"], 4), device=DEV)
        return {"case": case, "guide": g, "camera": sc.camera, "film": film, "seed": seed,
                "params": {"width": case["width"], "height": case["height"], "sampleCount": case["spp"],
                           "maxDepth": case["depth"]}}
    if kind == "train":
        sc = _scene("guiding", 0)
        g = gpu.GpuGuide(_tree(sc), seed=seed, batch=case["batch"])
        film = torch.zeros((180, 320, 4), device=DEV)
        for k in range(2):   # two collection passes fill the ring
            g.render(sc.camera, {"width": 320, "height": 180, "sampleCount": 2, "maxDepth": 12}, film,
                     gpu.GUIDE_GUIDED | gpu.GUIDE_COLLECT, seed=seed, sample_offset=2 * k)
        return {"case": case, "guide": g}
    ctx = gpu.Context()
    return {"case": case, "ctx": ctx, "film": _film(case, seed)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "host_rays":
        if case["any"]:
            return {"hit": state["acc"].intersect_any(state["org"], state["dir"], state["tmax"])}
        prim, t, u, v = state["acc"].intersect(state["org"], state["dir"], state["tmax"])
        return {"prim": prim, "t": t, "u": u, "v": v}
    if kind in ("rays", "build"):
        if kind == "build":
            state["acc"].construct()
        any_hit = case.get("any", False)
        out = state["out"]
        state["acc"].intersect_device(state["org"], state["dir"], out, any_hit=any_hit)
        got = {"hit": out} if any_hit else {"prim": out.view(torch.int32)[:, 1], "t": out[:, 0], "u": out[:, 2],
                                            "v": out[:, 3]}
        if kind == "build":
            info = state["acc"].info()
            got.update(nodes=int(info.wide_nodes), depth=int(info.depth), triangles=int(info.triangles),
                       bounds=np.array(info.bounds, np.float32))
        return got
    if kind == "render":
        integ, acc, params = state["integ"], state["acc"], state["params"]
        if case["host"]:
            film = integ.render(state["camera"], acc, params)
            st = integ.last_stats
        else:
            film = state["film"]
            film.zero_()
            st = integ.render_device(state["camera"], acc, params, film)
        return {"film": film, "paths": int(st.paths), "rays": int(st.rays_closest)}
    if kind == "batch":
        state["films"].zero_()
        _, st = state["batch"].run(state["films"])
        return {"films": state["films"], "paths": int(st.paths)}
    if kind == "guided":
        state["film"].zero_()
        st = state["guide"].render(state["camera"], state["params"], state["film"], gpu.GUIDE_GUIDED,
                                   seed=state["seed"])
        return {"film": state["film"], "paths": int(st.paths)}
    if kind == "train":
        loss = state["guide"].train(case["steps"])
        return {"params": state["guide"].params(), "loss": loss}
    fmt, param = FORMATS[case["format"]]
    return {"image": gpu.film_resolve(state["ctx"], state["film"], fmt, param)}


# ------------------------------------------------------------------------------ work
def _ray_flops(ntri):
    """A ray's unavoidable arithmetic: eight box tests on each level of an ideal 8-wide tree
    and two triangle tests."""
    levels = max(1.0, math.log(max(ntri, 8) / 2.0, 8))
    return levels * 8 * 14 + 2 * 45


def work(case):
    kind = case["kind"]
    if kind in ("host_rays", "rays"):
        ntri = 4 * 4 ** case["levels"]
        return {"bytes": case["rays"] * (32 + (4 if case["any"] else 16)) + 36 * ntri,
                "flops": case["rays"] * _ray_flops(ntri)}
    if kind == "build":
        # vertices, materials and lights in; leaf-order triangles and nodes out
        ntri = 4 * 4 ** case["size"] if case["scene"] == "sphere" else 4067 * case["size"]
        return {"bytes": ntri * (44 + 56 + 12), "flops": ntri * 300}
    if kind == "film":
        n = case["width"] * case["height"]
        per_out = {"rgbe": 4, "gamma": 3}.get(case["format"], 12)
        ops = {"rgbe": 20, "gamma": 60, "reinhard": 60, "drago": 120, "durand": 600}[case["format"]]
        return {"bytes": n * (16 + per_out), "flops": n * ops}
    if kind == "train":
        b, s = case["batch"], case["steps"]
        return {"bytes": s * (b * 64 + 4 * 11560 * 6), "flops": s * b * (22656 + 45312)}
    if kind == "batch":
        vs = scenes.batch_variants(case["renders"], seed=case["variants"])
        paths, pixels, ntri, vertices = sum(v.width * v.height * v.spp for v in vs), sum(v.width * v.height for v in vs), 36, 5
    else:
        pixels = case["width"] * case["height"]
        paths = pixels * case["spp"]
        name = "guiding" if kind == "guided" else case["scene"]
        ntri = {"mid": 2033674, "guiding": 2418}.get(name, 36)
        vertices = 1 if case.get("integrator") == "direct" else min(case["depth"], 5)
    # per path vertex: one closest-hit and about one shadow ray, and some 300 operations of
    # shading (and the network's where it is sampled)
    flops = paths * vertices * (2 * _ray_flops(ntri) + 300 + (22656 if kind == "guided" else 0))
    return {"bytes": pixels * 16 + 36 * ntri, "flops": flops}


# ------------------------------------------------------------------------------ exact
def _exact_rays(org, dirs, verts):
    """Closest hits by testing every triangle in 64 bits: t, u, v (0 where nothing is hit)."""
    V = torch.from_numpy(verts).to(DEV).double().reshape(-1, 3, 3)
    p0 = V[:, 0]
    e1, e2 = V[:, 1] - p0, V[:, 2] - p0
    o, d, tmax = org[:, :3].double(), dirs[:, :3].double(), dirs[:, 3].double()
    out = torch.zeros((o.shape[0], 3), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 24) // V.shape[0])
    for i in range(0, o.shape[0], step):
        D, O = d[i:i + step, None], o[i:i + step, None]
        pv = torch.linalg.cross(D.expand(-1, V.shape[0], -1), e2[None])
        det = (pv * e1).sum(-1)
        tv = O - p0
        u = (tv * pv).sum(-1) / det
        qv = torch.linalg.cross(tv, e1[None].expand_as(tv))
        v = (D * qv).sum(-1) / det
        t = (qv * e2).sum(-1) / det
        ok = (det.abs() >= 1e-12) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-12)
        ok &= t <= tmax[i:i + step, None]
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, k = t.min(1)
        hit = torch.isfinite(best)
        row = torch.stack([best, u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]], 1)
        out[i:i + step] = torch.where(hit[:, None], row, torch.zeros_like(row))
    return out


def _exact_film(case, seed):
    eps = 1.0e-12
    f = _film(case, seed).double()
    img = f[..., :3] / (f[..., 3:] + eps)
    weights = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=DEV)
    L = (img * weights).sum(-1)
    n = L.numel()
    mean = torch.exp(torch.log(L + eps).sum() / n)
    chroma = img / (L + eps)[..., None]
    p = FORMATS[case["format"]][1]
    if case["format"] == "reinhard":
        s = L.flatten().sort().values
        hi, lo = s[min(int(n * 0.99), n - 1)], s[min(int(n * 0.01), n - 1)]
        white = 1.5 * 2.0 ** (torch.log2(hi + eps) - torch.log2(lo + eps) - 5)
        Ls = p * L / mean
        return chroma * (Ls * (1.0 + Ls / (white * white)) / (1.0 + Ls))[..., None]
    if case["format"] == "drago":
        wa = mean / (1.0 + p - 0.85) ** 5.0
        top = L.max() / wa
        c1, c2 = math.log(p) / math.log(0.5), 1.0 / torch.log10(1.0 + top)
        return chroma * (c2 * torch.log1p(L / wa) / torch.log(2.0 + 8.0 * (L / wa / top) ** c1))[..., None]
    logL = torch.log10(L + 1.0e-6)
    sigma = max(case["width"], case["height"]) * 0.02
    dx = 1.0 + sigma / 0.4 * (logL[:, 1:] - logL[:, :-1]).abs()
    dy = 1.0 + sigma / 0.4 * (logL[1:] - logL[:-1]).abs()
    y = logL.clone()
    for i in range(20):
        a = math.exp(-math.sqrt(2.0) / (sigma * math.sqrt(3.0) * 2.0 ** (19 - i) / math.sqrt(4.0 ** 20 - 1.0)))
        if a == 0.0:
            break   # no feedback is left
        for lines, V in ((y.T, (a ** dx).T), (y, a ** dy)):
            for k in range(1, lines.shape[0]):
                lines[k] += V[k - 1] * (lines[k - 1] - lines[k])
            for k in range(lines.shape[0] - 2, -1, -1):
                lines[k] += V[k] * (lines[k + 1] - lines[k])
    base = torch.clamp(10.0 ** y - 1.0e-6, min=0.0)
    lb, ld = torch.log10(base + eps), torch.log10(L / (base + eps) + eps)
    cf = math.log(p) / (lb.max() - lb.min())
    return torch.clamp(chroma * (10.0 ** (lb * cf + ld - cf * lb.max()))[..., None], 0.0, 1.0)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("host_rays", "rays") and not case["any"] and case["rays"] * 4 * 4 ** case["levels"] <= 4e9:
        sc = _sphere(case["levels"])
        hit = _exact_rays(*_rays(case, seed, sc), sc.verts)
        return {"prim": None, "t": hit[:, 0], "u": hit[:, 1], "v": hit[:, 2]}
    if kind == "film" and case["format"] in ("reinhard", "drago", "durand"):
        return {"image": _exact_film(case, seed)}
    return None
