"""Closest hits among triangles at exactly one distance.

The walk keeps the first such triangle it meets, children nearest first and
children at one distance in the order in which its sorting network leaves them.
That is a property of the ray and the tree: neither the batch around a ray nor
the kernel that ends it may show.  The scenes are right triangles with power of
two legs in planes across the rays, at multiples of 1/64, so that every distance
and every product of the tests is exact and a walk over the host's tree in
Python gives the one right answer.
"""
import numpy as np
import pytest

from rise_b200 import raycaster, scenes

from risemesh_io import risemesh_bytes, soup_mesh

pytestmark = pytest.mark.gpu

RAYS = 512


def right_triangles(n, planes, seed):
    """n right triangles, coordinates multiples of 1/64, in the given z planes."""
    g = np.random.default_rng(seed)
    leg = 2.0 ** -g.integers(1, 4, (n, 2))
    o = np.stack([g.integers(0, 64, n) / 64 * (1 - leg[:, 0]), g.integers(0, 64, n) / 64 * (1 - leg[:, 1])], 1)
    o = np.round(o * 64) / 64
    z = np.asarray(planes, np.float64)[g.integers(0, len(planes), n)]
    tri = np.zeros((n, 3, 3), np.float32)
    tri[:, :, :2] = o[:, None]
    tri[:, 1, 0] += leg[:, 0]
    tri[:, 2, 1] += leg[:, 1]
    tri[:, :, 2] = z[:, None]
    flip = g.random(n) < 0.5
    tri[flip] = tri[flip][:, ::-1]
    return tri.reshape(n, 9)


def upward_rays(n, seed):
    """Rays along +z; x and y are odd multiples of 1/256, off every box plane."""
    g = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, 0] = (2 * g.integers(0, 128, n) + 1) / 256
    r[:, 1] = (2 * g.integers(0, 128, n) + 1) / 256
    r[:, 2] = -1.0
    r[:, 6] = 1.0
    r[:, 7] = np.inf
    return r


def ordered(children):
    """[(distance, child or None)] * 4 as the walk's network leaves them."""
    e = list(children)
    for i, j in ((0, 1), (2, 3), (0, 2), (1, 3), (1, 2)):
        if e[j][0] < e[i][0]:
            e[i], e[j] = e[j], e[i]
    return [c for _, c in e if c is not None]


def walk(tri, prims, nodes, ray):
    """The closest hit of a +z ray: the first triangle met at the least distance."""
    x, y, oz = (float(v) for v in ray[:3])
    best, found = np.inf, -1
    stack = [0]
    while stack:
        e = stack.pop()
        if isinstance(e, tuple):
            for p in prims[e[0]:e[0] + e[1]]:
                a, b, c = (tri[p, 3 * k:3 * k + 2].astype(np.float64) - (x, y) for k in range(3))
                w = [b[0] * c[1] - b[1] * c[0], c[0] * a[1] - c[1] * a[0], a[0] * b[1] - a[1] * b[0]]
                t = float(tri[p, 2]) - oz
                if (min(w) >= 0 or max(w) <= 0) and t < best:
                    best, found = t, int(p)
            continue
        n = nodes[e]
        kids = []
        for i in range(4):
            kid = (np.inf, None)
            if i < n["nchild"] and n["minx"][i] < x < n["maxx"][i] and n["miny"][i] < y < n["maxy"][i]:
                near, far = float(n["minz"][i] - ray[2]), float(n["maxz"][i] - ray[2])   # in FP32
                if near <= min(far, best):
                    first, count = int(n["child"][i]), int(n["count"][i])
                    kid = (near, (first, count) if count else first)
            kids.append(kid)
        stack += ordered(kids)[::-1]
    return found


def cast(rc, rays):
    import torch
    d = torch.from_numpy(rays).cuda()
    out = torch.empty(len(rays), 4, device="cuda")
    rc.cast_rays_device(d.data_ptr(), out.data_ptr(), len(rays), torch.cuda.current_stream().cuda_stream)
    return out.cpu().numpy().view(raycaster.HIT_DTYPE)[:, 0]


def many_rays(ctx):
    """More rays than the kernels whose warps end their last rays together take."""
    import torch
    return 4096 * torch.cuda.get_device_properties(ctx.device).multi_processor_count + 4097


PLANES = ([0.25], [0.25, 0.5, 0.75])


@pytest.mark.parametrize("planes", PLANES)
@pytest.mark.parametrize("layout", ["f32", "f16"])
def test_children_at_one_distance_keep_their_order(layout, planes):
    tri = right_triangles(400, planes, 3)
    _, prims, nodes = raycaster.build_host_bvh(tri)
    rays = upward_rays(RAYS, 4)
    want = np.array([walk(tri, prims, nodes, r) for r in rays])
    assert (want >= 0).mean() > 0.8
    with raycaster.Context(0) as ctx:
        s = raycaster.Scene(ctx)
        s.add_triangles(tri)
        s.commit(layout)
        n = many_rays(ctx)
        got = cast(raycaster.RayCaster(s), np.tile(rays, (n // RAYS + 1, 1))[:n])["prim"]
        assert np.array_equal(got, np.tile(want, n // RAYS + 1)[:n])
        s.close()


def soup_twice():
    tri = scenes.soup_triangles(10_000, seed=3)
    return np.concatenate([tri, tri])[np.random.default_rng(7).permutation(20_000)], None


def long_leaves():
    """Leaves of twelve coincident triangles, in both windings."""
    tri = scenes.soup_triangles(3_000, seed=3)
    both = np.concatenate([tri, tri[:, [3, 4, 5, 0, 1, 2, 6, 7, 8]]] * 6)
    return both[np.random.default_rng(7).permutation(len(both))], None


def merged_meshes():
    tri = scenes.soup_triangles(6_000, seed=3)
    return None, [tri[:4000], tri[2000:], tri[1000:5000]]


def deep_twice():
    """A tree deeper than the shared-memory stack."""
    tri = scenes.nested_clusters()
    return np.concatenate([tri, tri]), None


@pytest.mark.parametrize("make,layout", [
    (m, v) for m in (soup_twice, long_leaves, merged_meshes, deep_twice) for v in ("f32", "q8", "f16", "w8")
    if not (m is deep_twice and v == "w8")])   # the eight-wide layout refuses its leaves
def test_coincident_triangles_answer_alike_in_every_batch(make, layout):
    tri, parts = make()
    with raycaster.Context(0) as ctx:
        s = raycaster.Scene(ctx)
        for p in parts or []:
            nodes2, prims, _ = raycaster.build_host_bvh(p)
            pts, idx = soup_mesh(p)
            s.add_risemesh(raycaster.RiseMesh(risemesh_bytes(pts, idx, nodes2=nodes2, prims=prims)))
        if tri is not None:
            s.add_triangles(tri)
        s.commit(layout)
        rc = raycaster.RayCaster(s)
        n = many_rays(ctx)
        rays = scenes.cluster_rays(tri, n, 5) if make is deep_twice else scenes.sphere_rays(n, 5)
        hits = cast(rc, rays)
        assert (hits["prim"] >= 0).mean() > 0.05
        for k in (1, 5, 64, 4095, 20_000, 100_003, n - 4097):
            for repeat in range(10 if k > 20_000 else 2):
                assert cast(rc, rays[:k]).tobytes() == hits[:k].tobytes(), (k, repeat)
        s.close()


@pytest.mark.parametrize("planes", PLANES)
@pytest.mark.parametrize("layout", ["f32", "f16"])
def test_small_batches_keep_the_first_triangle_met(layout, planes):
    tri = right_triangles(400, planes, 3)
    _, prims, nodes = raycaster.build_host_bvh(tri)
    rays = upward_rays(RAYS, 4)
    want = np.array([walk(tri, prims, nodes, r) for r in rays])
    with raycaster.Context(0) as ctx:
        s = raycaster.Scene(ctx)
        s.add_triangles(tri)
        s.commit(layout)
        rc = raycaster.RayCaster(s)
        for n in (1, 3, 64, RAYS):
            for k in range(0, RAYS, max(n, 32)):
                assert np.array_equal(cast(rc, rays[k:k + n])["prim"], want[k:k + n]), (n, k)
        s.close()


def test_coincident_meshes_render_alike_alone_and_in_a_batch():
    """Two meshes of different materials in one place: a path's hit, and so the
    image, is the same from run to run and among other scenes' paths.  Alone
    360,000 paths start at once, in the engine 16,384: other walks end them."""
    from rise_b200 import pathtracer
    descs = []
    for k in range(2):
        d = scenes.spheres_scene(grid=32 + 8 * k, n_spheres=4, sphere_tris=600, width=200, height=150, seed=3 + k, max_depth=6)
        tri, meshes = d.tri9, list(d.meshes)
        for first, count, mat, ds in meshes[:3]:
            d.add_mesh(tri[first:first + count], (mat + 1) % len(d.materials), ds)
        descs.append(d)
    with raycaster.Context(0) as ctx:
        devs = [pathtracer.upload_scene(ctx, d) for d in descs]

        def job(k):
            return pathtracer.SpectralRasterizer(ctx, descs[k], scene=devs[k])

        films = []
        for k in range(2):
            for _ in range(3):
                r = job(k)
                r.rasterize_scene(12)
                films.append((k, r.film()))
                r.close()
        for use_graph in (False, True):
            eng = pathtracer.Engine(ctx, 1 << 14)
            jobs = [job(0), job(1)]
            eng.render(jobs, [12, 12], use_graph=use_graph)
            films += [(k, j.film()) for k, j in enumerate(jobs)]
            for j in jobs:
                j.close()
            eng.close()
        first = {0: films[0][1], 1: films[3][1]}
        for n, (k, f) in enumerate(films):
            assert np.allclose(f, first[k], rtol=1e-5, atol=1e-6), n
        for d in devs:
            d.close()
