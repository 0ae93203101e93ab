"""The kernels' dispatch rules on the GPU: calls on both sides of a rule give the same
results."""
import pytest

from spica_gb300 import GpuBVHAccel, scenes

pytestmark = pytest.mark.gpu


def _device_rays(n, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    org = torch.zeros((n, 4), device="cuda")
    dirs = torch.zeros((n, 4), device="cuda")
    org[:, :3] = 2.4 * torch.rand((n, 3), device="cuda", generator=g) - 1.2
    dirs[:, :3] = torch.randn((n, 3), device="cuda", generator=g)
    dirs[:, :3] /= dirs[:, :3].norm(dim=1, keepdim=True)
    dirs[:, 3] = 1.0e32
    return org, dirs


@pytest.mark.parametrize("levels", [4, 5])            # trees below and above 512 wide nodes
@pytest.mark.parametrize("rays", [(1 << 21) - 1, 1 << 21, (1 << 21) + 33])
def test_split_traversal_matches_whole_steps(gpulib, levels, rays):
    """Closest hits of 2^21 rays and more on larger trees are traced in the split form
    (the same order of triangle tests per ray), smaller batches in whole steps:
    every hit record is the same bit for bit."""
    import torch
    acc = GpuBVHAccel(scenes.displaced_sphere(levels=levels, seed=1)).construct()
    assert (acc.info().wide_nodes >= 512) == (levels == 5)
    org, dirs = _device_rays(rays, 7)
    out = torch.full((rays, 4), -1.0, device="cuda")
    acc.intersect_device(org, dirs, out)
    parts = torch.full((rays, 4), -1.0, device="cuda")
    for a in range(0, rays, 1 << 20):
        acc.intersect_device(org[a:a + (1 << 20)], dirs[a:a + (1 << 20)], parts[a:a + (1 << 20)])
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int32), parts.view(torch.int32))
    assert 0.1 < (out.view(torch.int32)[:, 1] >= 0).float().mean().item() < 1.0


ROOMS = {"box": scenes.box_room, "material": scenes.material_room, "conductor": scenes.conductor_room}


@pytest.mark.parametrize("room, width, height, spp, depth, integrator", [
    ("box", 1, 1, 1, 0, "path"),             # one path, emission only
    ("box", 33, 17, 1, 64, "path"),          # one sample; deeper than the iterations between two looks
    ("material", 64, 48, 5, 17, "path"),     # all classes; odd samples; one iteration past a look
    ("conductor", 40, 30, 3, 16, "path"),
    ("box", 512, 512, 2, 3, "path"),         # 2^19 paths: the last of one class in one lane
    ("box", 512, 513, 2, 3, "path"),
    ("box", 1024, 1025, 1, 3, "path"),       # one sample cannot be shared
    ("material", 512, 512, 4, 3, "path"),    # 2^20 paths: the last in one lane
    ("material", 512, 513, 5, 3, "path"),    # two lanes, uneven shares
    ("material", 65, 31, 4, 5, "direct"),
])
def test_one_pass_render_matches_pass_by_pass(gpulib, room, width, height, spp, depth, integrator):
    """A render whose paths fit the pools at once takes one pass over depth + 1 iterations; the
    pass-by-pass wavefront draws the same samples and traces the same rays, so the films agree up
    to the order of their additions (1e-5 relative, and 1e-6 of the largest value for values
    that cancel small terms, on 99.9 % of values, as for the refilling loop)."""
    import torch
    from spica_gb300 import Context, GpuDirectLightingIntegrator, GpuPathIntegrator
    sc = ROOMS[room](width=width, height=height)
    params = {"width": width, "height": height, "maxDepth": depth, "sampleCount": spp}
    got = []
    for wavefront in (0, 1):
        acc = GpuBVHAccel(sc, ctx=Context(0, wavefront=wavefront)).construct()
        integ = (GpuPathIntegrator if integrator == "path" else GpuDirectLightingIntegrator)(seed=5)
        film = torch.zeros((height, width, 4), device="cuda")
        st = integ.render_device(sc.camera, acc, params, film, sample_offset=2)
        got.append((film.cpu(), st.paths, st.rays_closest, st.rays_shadow))
    (a, *sa), (b, *sb) = got
    assert sa == sb and sa[0] == width * height * spp
    assert torch.equal(a[..., 3], b[..., 3]) and bool((a[..., 3] == spp).all())
    x, y = a[..., :3], b[..., :3]
    close = (x - y).abs() <= 1e-5 * y.abs() + 1e-6 * float(y.abs().max())
    assert close.float().mean() > 0.999


@pytest.mark.parametrize("triangles", [1, 2, 3, 4, 5, 31, 32, 33, 65, 1023, 1025, 2047, 2048, 2049, 2050, 5000, 20000])
def test_build_sizes(gpulib, port, triangles):
    """Trees on both sides of the build's steps (one block for the last 2048 clusters, rounds of
    1024-cluster blocks before): every triangle is placed, and the closest hits of random rays
    are the oracle's under the parity rules of tests/parity.py."""
    import numpy as np
    from parity import classify_closest
    rng = np.random.default_rng(triangles)
    c = rng.random((triangles, 1, 3)) * 2 - 1
    size = np.where(rng.random((triangles, 1, 1)) < 0.02, 1.0, 1.5 / np.sqrt(triangles))
    sc = scenes.Scene(verts=(c + size * (rng.random((triangles, 3, 3)) - 0.5)).reshape(-1, 9).astype(np.float32),
                      tri_mat=np.zeros(triangles, np.int32), materials=np.array([scenes.lambert(0.5, 0.5, 0.5)]))
    acc = GpuBVHAccel(sc).construct()
    info = acc.info()
    assert info.triangles == triangles and 1 <= info.wide_nodes <= max(1, triangles - 1) and info.depth >= 1
    lo, hi = acc.worldBound()
    v = sc.verts.reshape(-1, 3)
    np.testing.assert_array_equal(np.array([lo, hi], np.float32), [v.min(0), v.max(0)])
    target = sc.verts.reshape(-1, 3, 3)[rng.integers(0, triangles, 4000)].mean(1)
    org = (2.5 * rng.normal(size=(4000, 3))).astype(np.float32)
    d = target - org
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    prim, t, _, _ = acc.intersect(org, d)
    pr, tr = port.scene(sc).trace(org.astype(np.float64), d.astype(np.float64))
    r = classify_closest(sc.verts, org, d, prim, t, pr, tr)
    assert r["fail"] == 0 and r["t_fail"] == 0, r
    assert (prim >= 0).mean() > 0.9


def _one_class_room(cls, width, height):
    sc = ROOMS["material" if cls == 2 else "box" if cls == 0 else "conductor"](width=width, height=height)
    if cls == 1:      # rough conductors alone
        sc.materials = sc.materials[-2:]
        sc.tri_mat = (sc.tri_mat % 2).astype(sc.tri_mat.dtype)
    elif cls == 2:    # plastic alone
        sc.materials = sc.materials[-1:]
        sc.tri_mat = 0 * sc.tri_mat
    return sc


@pytest.mark.parametrize("cls", [0, 1, 2])
@pytest.mark.parametrize("width, height, spp", [(64, 48, 3), (3001, 3000, 2)])   # one pass; the refilling loop
def test_one_class_scene_matches_pass_by_pass(gpulib, cls, width, height, spp):
    """Scenes of one shading class are shaded out of the pool itself, rays and continuations in
    two pools that change places; rays leave the rooms through their open side, so there are
    rows without a hit.  Same samples and rays as the pass-by-pass wavefront, films equal up to
    the order of their additions (the bounds of test_one_pass_render_matches_pass_by_pass)."""
    import torch
    from spica_gb300 import Context, GpuPathIntegrator
    sc = _one_class_room(cls, width, height)
    params = {"width": width, "height": height, "maxDepth": 5, "sampleCount": spp}
    got = []
    for wavefront in (0, 1):
        acc = GpuBVHAccel(sc, ctx=Context(0, pass_lanes=1, wavefront=wavefront)).construct()
        film = torch.zeros((height, width, 4), device="cuda")
        st = GpuPathIntegrator(seed=8).render_device(sc.camera, acc, params, film)
        got.append((film, st.paths, st.rays_closest, st.rays_shadow))
        del acc
    (a, *sa), (b, *sb) = got
    assert sa == sb and sa[0] == width * height * spp
    assert torch.equal(a[..., 3], b[..., 3])
    x, y = a[..., :3], b[..., :3]
    close = (x - y).abs() <= 1e-5 * y.abs() + 1e-6 * float(y.abs().max())
    assert close.float().mean() > 0.999


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("rays", [1, 33, 4096, 4097, 65536, 65537, 155647, 155648, 155649])
def test_ray_batch_routes_agree(gpulib, any_hit, rays):
    """Host batches up to 65,536 rays are read from and written to pinned host memory, larger ones
    copied; batches of at most a resident grid's lanes (152 SMs x 8 blocks x 128) take no ray
    counter.  Host and device entry points give the same records as one 2^18-ray device batch."""
    import numpy as np
    import torch
    acc = GpuBVHAccel(scenes.displaced_sphere(levels=4, seed=3)).construct()
    org, dirs = _device_rays(1 << 18, 11)
    shape = (1 << 18,) if any_hit else (1 << 18, 4)
    if any_hit:
        dirs[:, 3] = 0.8
    whole = torch.zeros(shape, dtype=torch.int32, device="cuda")
    acc.intersect_device(org, dirs, whole, any_hit=any_hit)
    part = torch.full((rays, *shape[1:]), -7, dtype=torch.int32, device="cuda")
    for _ in range(2):   # again over the same buffers
        acc.intersect_device(org[:rays], dirs[:rays], part, any_hit=any_hit)
    torch.cuda.synchronize()
    assert torch.equal(part, whole[:rays])
    o, d = org[:rays].cpu().numpy(), dirs[:rays].cpu().numpy()
    want = whole[:rays].cpu().numpy()
    for _ in range(2):
        if any_hit:
            np.testing.assert_array_equal(acc.intersect_any(o[:, :3], d[:, :3], d[:, 3]), want.astype(bool))
        else:
            prim, t, u, v = acc.intersect(o[:, :3], d[:, :3], d[:, 3])
            np.testing.assert_array_equal(prim, want[:, 1])
            for got, k in ((t, 0), (u, 2), (v, 3)):
                np.testing.assert_array_equal(got.view(np.int32), want[:, k])


def test_host_films_of_changing_size(gpulib):
    """Host renders through the context's kept film buffer, growing and shrinking, add to the
    caller's film as the device entry point adds to a device film (the order of the additions of
    four samples: 1e-6 relative)."""
    import numpy as np
    import torch
    from spica_gb300 import GpuPathIntegrator
    sc = scenes.box_room(width=32, height=32)
    acc = GpuBVHAccel(sc).construct()
    integ = GpuPathIntegrator(seed=4)
    for w, h in ((16, 8), (64, 48), (5, 3), (64, 49)):
        p = {"width": w, "height": h, "maxDepth": 4, "sampleCount": 4}
        host = integ.render(sc.camera, acc, p, film=np.full((h, w, 4), 0.5, np.float32))
        dev = torch.full((h, w, 4), 0.5, device="cuda")
        integ.render_device(sc.camera, acc, p, dev)
        np.testing.assert_allclose(host, dev.cpu().numpy(), rtol=1e-6, atol=1e-6)
        assert np.all(host[..., 3] == 4.5)
