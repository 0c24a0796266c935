"""Timed cases: batched ray casts and spectral renders through the package's public entry points.

Two families, as a program uses them:

* casts: a committed scene and a batch of rays, closest hit or occlusion, with the rays on the
  device (RayCaster.cast_rays_device / cast_shadow_rays_device on the caller's stream) or in host
  arrays (RayCaster.cast_rays / cast_shadow_rays);
* renders: a resident scene and one image of it, progressive (a kept SpectralRasterizer that adds
  samples), one-shot (a job made, rendered, read and closed), adaptive, or several images at once
  in a shared Engine.

`prepare` builds and commits the scene (a user keeps it resident) and makes the rays; `run` is one
call and its whole result.
"""
import math

import numpy as np
import torch

from rise_b200 import pathtracer, raycaster, scenes

LAYOUTS = ("f32", "q8", "f16")
MAX_RAYS = 4_194_304
MAX_TRIANGLES = 1_000_000


def listed():
    return [
        # A handful of picking / probe rays per frame: launch latency only.
        {"name": "closest_64", "op": "cast", "geometry": "soup", "query": "closest", "where": "device",
         "layout": "f32", "triangles": 2_000, "rays": 64},
        # One light's occlusion queries for a small tile of shading points.
        {"name": "shadow_4k", "op": "cast", "geometry": "soup", "query": "shadow", "where": "device",
         "layout": "q8", "triangles": 30_000, "rays": 4_095},
        # One bounce of a small image: an ordinary batch of incoherent rays, odd size.
        {"name": "closest_100k", "op": "cast", "geometry": "soup", "query": "closest", "where": "device",
         "layout": "f16", "triangles": 300_000, "rays": 100_003},
        # Primary visibility of a 1024x768 image of a landscape: coherent rays, exact FP32 boxes.
        {"name": "camera_786k", "op": "cast", "geometry": "terrain", "query": "closest", "where": "device",
         "layout": "f32", "triangles": 400_000, "rays": 786_432},
        # Shadow rays of a large wavefront.
        {"name": "shadow_2m", "op": "cast", "geometry": "soup", "query": "shadow", "where": "device",
         "layout": "f16", "triangles": 1_000_000, "rays": 2_000_003},
        # The ray-cast microbenchmark at full size (bench.py).
        {"name": "closest_4m", "op": "cast", "geometry": "soup", "query": "closest", "where": "device",
         "layout": "f16", "triangles": 1_000_000, "rays": 4_194_304},
        # Rays and hits in host memory: a CPU renderer handing over one batch.
        {"name": "host_closest_250k", "op": "cast", "geometry": "soup", "query": "closest", "where": "host",
         "layout": "q8", "triangles": 100_000, "rays": 250_001},
        # A thumbnail of a small scene: job made, rendered, read back, closed.
        {"name": "render_thumb", "op": "render", "mode": "oneshot", "scene": "spheres", "triangles": 20_000,
         "width": 120, "height": 80, "spp": 4, "layout": "f32", "sampler": 2, "filter": 0, "nee": 1},
        # The spectral Cornell box (bench.py's C1 size), progressive passes of 16 spp.
        {"name": "render_cornell", "op": "render", "mode": "progressive", "scene": "cornell", "triangles": 32,
         "width": 256, "height": 256, "spp": 16, "layout": "f32", "sampler": 2, "filter": 0, "nee": 1},
        # A large scene of mixed materials (heightfield, GGX and glass spheres, sky).
        {"name": "render_spheres", "op": "render", "mode": "progressive", "scene": "spheres", "triangles": 800_000,
         "width": 1024, "height": 1024, "spp": 8, "layout": "f16", "sampler": 0, "filter": 0, "nee": 1},
        # Adaptive sampling into a Gaussian film, shared light samples.
        {"name": "render_adaptive", "op": "render", "mode": "adaptive", "scene": "cornell", "triangles": 32,
         "width": 200, "height": 150, "spp": 64, "layout": "f16", "sampler": 2, "filter": 1, "nee": 0},
        # Several small requests of different scenes in one engine (a render server's batch).
        {"name": "render_batch", "op": "render", "mode": "batch", "scene": "spheres", "triangles": 60_000,
         "width": 128, "height": 128, "spp": 8, "layout": "q8", "sampler": 0, "filter": 0, "nee": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.55:
        geometry = rng.choice(("soup", "soup", "terrain"))
        return {"op": "cast", "geometry": geometry, "query": rng.choice(("closest", "shadow")),
                "where": rng.choice(("device", "device", "host")), "layout": rng.choice(LAYOUTS),
                "triangles": _log(rng, 500, MAX_TRIANGLES), "rays": _log(rng, 16, MAX_RAYS)}
    mode = rng.choice(("progressive", "oneshot", "adaptive", "batch"))
    return {"op": "render", "mode": mode, "scene": rng.choice(("cornell", "spheres")),
            "triangles": _log(rng, 5_000, 800_000 if mode != "batch" else 100_000),
            "width": _log(rng, 32, 640 if mode != "batch" else 200),
            "height": _log(rng, 32, 640 if mode != "batch" else 200),
            "spp": 32 + _log(rng, 1, 32) if mode == "adaptive" else _log(rng, 1, 16),
            "layout": rng.choice(LAYOUTS), "sampler": rng.choice((0, 1, 2)), "filter": rng.choice((0, 0, 1)),
            "nee": rng.choice((0, 1, 1))}


class State:
    """What a program holds between calls; gives its device memory back when dropped."""

    def __init__(self):
        self.ctx = raycaster.Context(0)
        self.scenes, self.jobs, self.engine = [], [], None

    def __del__(self):
        if self.engine is not None:
            self.engine.close()
        for j in self.jobs:
            j.close()
        for s in self.scenes:
            s.close()
        self.ctx.close()


def _terrain(n_tri, seed):
    return scenes.batch_scene({"n_tri": n_tri, "res": 256, "max_depth": 8, "seed": seed})


def _unit(x):
    return x / x.norm(dim=1, keepdim=True)


def _sphere_rays(n, shadow, gen):
    """Rays from a radius-2 sphere around the cube's centre to uniform targets in the unit cube."""
    o = 0.5 + 2.0 * _unit(torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64))
    d = torch.rand(n, 3, generator=gen, device="cuda", dtype=torch.float64) - o
    dist = d.norm(dim=1, keepdim=True)
    return _rays(o, d / dist, dist if shadow else torch.full_like(dist, math.inf))


def _camera_rays(n, shadow, gen):
    """Jittered camera rays over a 4:3 raster in row order, or shadow rays from points above the
    terrain to a small light above it."""
    if shadow:
        u = torch.rand(n, 3, generator=gen, device="cuda", dtype=torch.float64)
        o = u * torch.tensor([1.0, 0.05, 1.0], device="cuda", dtype=torch.float64) + \
            torch.tensor([0.0, 0.1, 0.0], device="cuda", dtype=torch.float64)
        v = torch.rand(n, 3, generator=gen, device="cuda", dtype=torch.float64)
        tgt = v * torch.tensor([0.3, 0.0, 0.3], device="cuda", dtype=torch.float64) + \
            torch.tensor([0.35, 1.19, 0.35], device="cuda", dtype=torch.float64)
        d = tgt - o
        dist = d.norm(dim=1, keepdim=True)
        return _rays(o, d / dist, dist)
    w = max(1, int(math.sqrt(n * 4.0 / 3.0)))
    h = -(-n // w)
    i = torch.arange(n, device="cuda")
    jit = torch.rand(n, 2, generator=gen, device="cuda", dtype=torch.float64)
    sx = 2.0 * ((i % w).double() + jit[:, 0]) / w - 1.0
    sy = 1.0 - 2.0 * ((i // w).double() + jit[:, 1]) / h
    pos = torch.tensor([0.5, 0.55, -0.45], device="cuda", dtype=torch.float64)
    fwd = torch.tensor([0.0, -0.55, 1.0], device="cuda", dtype=torch.float64)
    fwd = fwd / fwd.norm()
    right = torch.tensor([1.0, 0.0, 0.0], device="cuda", dtype=torch.float64)
    up = torch.linalg.cross(fwd, right)
    d = _unit(fwd + 0.55 * sx[:, None] * right + 0.41 * sy[:, None] * up)
    return _rays(pos.expand(n, 3), d, torch.full((n, 1), math.inf, device="cuda", dtype=torch.float64))


def _rays(o, d, tmax):
    return torch.cat([o, torch.zeros_like(tmax), d, tmax], dim=1).float().contiguous()


def _cast_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["geometry"] == "soup":
        tri9 = scenes.soup_triangles(case["triangles"], seed)
        rays = _sphere_rays(case["rays"], case["query"] == "shadow", gen)
    else:
        tri9 = _terrain(case["triangles"], seed % 100_000).tri9
        rays = _camera_rays(case["rays"], case["query"] == "shadow", gen)
    return tri9, rays


def _render_desc(case, seed):
    if case["scene"] == "cornell":
        d = scenes.cornell_box(width=case["width"], height=case["height"])
    else:
        d = _terrain(case["triangles"], seed % 100_000)
    st = d.settings
    st.width, st.height = case["width"], case["height"]
    st.seed = seed & 0x7fffffff
    st.sampler, st.filter, st.nee_per_lambda = case["sampler"], case["filter"], case["nee"]
    if case["mode"] == "adaptive":
        st.adaptive_max_spp, st.adaptive_threshold = case["spp"], 0.1
    return d


def prepare(case, seed):
    s = State()
    s.case = case
    if case["op"] == "cast":
        tri9, rays = _cast_inputs(case, seed)
        scene = raycaster.Scene(s.ctx)
        s.scenes.append(scene)
        scene.add_triangles(tri9)
        scene.commit(case["layout"])
        s.caster = raycaster.RayCaster(scene)
        n = case["rays"]
        if case["where"] == "host":
            s.rays = rays.cpu().numpy()
        else:
            s.rays = rays
            s.out = torch.empty(n, 4, device="cuda") if case["query"] == "closest" else \
                torch.empty(n, dtype=torch.uint8, device="cuda")
        return s
    # A batch is four scenes whose sizes differ by up to eight, twice each at different resolutions.
    for k in range(4 if case["mode"] == "batch" else 1):
        sub = dict(case, triangles=max(500, case["triangles"] >> k))
        desc = _render_desc(sub, seed + 101 * k)
        scene = pathtracer.upload_scene(s.ctx, desc, case["layout"])
        s.scenes.append(scene)
        if case["mode"] == "oneshot" or case["mode"] == "adaptive":
            s.desc = desc
        elif case["mode"] == "progressive":
            s.jobs.append(pathtracer.SpectralRasterizer(s.ctx, desc, scene=scene))
        else:
            for j in range(2):
                st = scenes.RenderSettings(**{**desc.settings.__dict__, "width": max(16, case["width"] >> j),
                                              "seed": desc.settings.seed + j})
                s.jobs.append(pathtracer.SpectralRasterizer(s.ctx, desc, scene=scene, settings=st))
    if case["mode"] == "batch":
        s.engine = pathtracer.Engine(s.ctx, 1 << 18)
    return s


def run(s):
    case = s.case
    if case["op"] == "cast":
        if case["where"] == "host":
            if case["query"] == "shadow":
                return s.caster.cast_shadow_rays(s.rays)
            h = s.caster.cast_rays(s.rays)
            return {"t": h["t"], "prim": h["prim"], "a": h["a"], "b": h["b"]}
        stream = torch.cuda.current_stream().cuda_stream
        if case["query"] == "shadow":
            s.caster.cast_shadow_rays_device(s.rays.data_ptr(), s.out.data_ptr(), case["rays"], stream)
            return s.out
        s.caster.cast_rays_device(s.rays.data_ptr(), s.out.data_ptr(), case["rays"], stream)
        return {"t": s.out[:, 0], "prim": s.out[:, 1].view(torch.int32), "a": s.out[:, 2], "b": s.out[:, 3]}
    mode = case["mode"]
    if mode == "progressive":
        s.jobs[0].rasterize_scene(case["spp"])
        return s.jobs[0].film()
    if mode == "batch":
        # Uneven requests: the second image of each scene takes twice the samples.
        s.engine.render(s.jobs, [case["spp"] << (k & 1) for k in range(len(s.jobs))])
        return [j.film() for j in s.jobs]
    r = pathtracer.SpectralRasterizer(s.ctx, s.desc, scene=s.scenes[0])
    try:
        if mode == "oneshot":
            r.rasterize_scene(case["spp"])
            return {"xyz": r.film(), "rgb": r.rgb()}
        # The first convergence test comes at 32 samples; the rest go to pixels still noisy.
        r.rasterize_scene(32)
        r.rasterize_scene(case["spp"] - 32)
        return {"xyz": r.film(), "samples": r.sample_counts().view(np.int32)}
    finally:
        r.close()


def work(case):
    # A ray descends at least one root-to-leaf path of slab tests (14 flops each) and tests the
    # triangle it hits (about 60); it is read (32 bytes) and its answer written.
    ray_flops = 60 + 14 * math.log2(max(case["triangles"], 2))
    if case["op"] == "cast":
        n = case["rays"]
        out = 16 if case["query"] == "closest" else 1
        return {"bytes": n * (32 + out) + 36 * min(n, case["triangles"]), "flops": n * ray_flops}
    npix, tri = case["width"] * case["height"], case["triangles"]
    samples = npix * case["spp"]
    if case["mode"] == "adaptive":
        samples = npix * 32
    if case["mode"] == "batch":
        # Four scenes of n, n/2, n/4, n/8 triangles, each at full and half width (twice the samples).
        tri, npix, samples = tri * 15 / 8, 4 * npix * 1.5, 4 * npix * 2 * case["spp"]
    # About four path vertices a sample, each one extended ray, one or four light rays and about
    # 300 flops of shading; the scene's vertices are read once and the image written once.
    rays = 4 * (1 + (4 if case["nee"] else 1) * 0.6)
    return {"bytes": 36 * min(tri, samples) + 12 * npix, "flops": samples * (rays * ray_flops + 4 * 300)}


def exact(case, seed):
    """Closest hits in 64 bits over all ray-triangle pairs (a line-versus-edge sign test on Pluecker
    coordinates); occlusion flags are whole values and a path-traced image has no value of its own."""
    if case["op"] != "cast" or case["query"] != "closest" or case["rays"] * case["triangles"] > 4e10:
        return None
    tri9, rays = _cast_inputs(case, seed)
    tri = torch.from_numpy(tri9).to("cuda").double().view(-1, 3, 3)
    rays = rays.double()
    v = [tri[:, k] for k in range(3)]
    cross = torch.linalg.cross
    # Edge lines of the triangles, opposite vertex 0, 1, 2, and their planes.
    edge = [(v[(k + 2) % 3] - v[(k + 1) % 3], cross(v[(k + 1) % 3], v[(k + 2) % 3])) for k in range(3)]
    normal = cross(v[1] - v[0], v[2] - v[0])
    offset = (normal * v[0]).sum(1)
    n, m = len(rays), len(tri)
    t = torch.full((n,), math.inf, device="cuda", dtype=torch.float64)
    a, b = torch.zeros_like(t), torch.zeros_like(t)
    tmin, tmax = rays[:, 3], rays[:, 7]
    step_n, step_m = min(n, 8192), min(m, 16384)
    for i in range(0, n, step_n):
        o, d = rays[i:i + step_n, 0:3], rays[i:i + step_n, 4:7]
        line = torch.cat([d, cross(o, d)], dim=1)
        lo, hi = tmin[i:i + step_n, None], tmax[i:i + step_n, None]
        for j in range(0, m, step_m):
            # w[k]: side of the ray's line seen from the edge opposite vertex k.
            w = [line @ torch.cat([e[1][j:j + step_m], e[0][j:j + step_m]], dim=1).T for e in edge]
            det = w[0] + w[1] + w[2]
            nd = d @ normal[j:j + step_m].T
            tt = (offset[j:j + step_m] - o @ normal[j:j + step_m].T) / nd
            up = (w[0] >= 0) & (w[1] >= 0) & (w[2] >= 0)
            down = (w[0] <= 0) & (w[1] <= 0) & (w[2] <= 0)
            ok = (up | down) & (det.abs() >= 1e-12) & (tt > lo) & (tt < hi)
            best, at = torch.where(ok, tt, math.inf).min(dim=1)
            pick = lambda x: x.gather(1, at[:, None])[:, 0]  # noqa: E731
            near = best < t[i:i + step_n]
            t[i:i + step_n] = torch.where(near, best, t[i:i + step_n])
            a[i:i + step_n] = torch.where(near, pick(w[1]) / pick(det), a[i:i + step_n])
            b[i:i + step_n] = torch.where(near, pick(w[2]) / pick(det), b[i:i + step_n])
    hit = torch.isfinite(t)
    return {"t": torch.where(hit, t, -1.0), "prim": None, "a": torch.where(hit, a, 0.0),
            "b": torch.where(hit, b, 0.0)}
