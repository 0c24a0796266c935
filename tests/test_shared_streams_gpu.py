"""Host casts between the steps of an engine of the same context.

Renders run parts of an iteration on the streams and events of the host-cast
pipeline; each call leaves them idle for the other.
"""
import numpy as np
import pytest

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [False, True])
def test_casts_between_steps_change_nothing(use_graph):
    tri, n = scenes.soup_triangles(20_000, seed=3), 200_001
    rays, srays = scenes.sphere_rays(n, 3), scenes.sphere_rays(n, 4, shadow=True)
    desc = scenes.spheres_scene(grid=48, n_spheres=6, sphere_tris=600, width=96, height=64, max_depth=8)
    with raycaster.Context(0) as ctx:
        soup = raycaster.Scene(ctx)
        soup.add_triangles(tri)
        soup.commit("q8")
        rc = raycaster.RayCaster(soup)
        hits, occ = rc.cast_rays(rays).tobytes(), rc.cast_shadow_rays(srays).tobytes()
        scene = pathtracer.upload_scene(ctx, desc)
        alone = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
        alone.rasterize_scene(24)
        r = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
        eng = pathtracer.Engine(ctx, 1 << 14)
        eng.submit(r, 24)
        casts = 0
        while eng.progress(r)[0] < eng.progress(r)[1]:
            eng.step(2, use_graph=use_graph)
            assert rc.cast_rays(rays).tobytes() == hits
            assert rc.cast_shadow_rays(srays).tobytes() == occ
            casts += 1
            assert casts < 1000
        eng.retire(r)
        assert casts > 3 and np.allclose(r.film(), alone.film(), rtol=1e-5, atol=1e-7)
        for x in (r, alone):
            x.close()
        eng.close()
        for s in (soup, scene):
            s.close()
