"""A kept engine's captured graph and scenes that come and go.

A capture holds the pointers of the scene that all jobs share.  A new scene is
often made at the address of a destroyed one; it must not be taken for that.
"""
import numpy as np
import pytest

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu


def test_new_scene_in_an_old_ones_place_is_captured_anew():
    descs = [scenes.cornell_box(32, 24), scenes.spheres_scene(grid=16, n_spheres=2, sphere_tris=200, width=32, height=24),
             scenes.spheres_scene(grid=24, n_spheres=3, sphere_tris=400, width=32, height=24, seed=5)]
    with raycaster.Context(0) as ctx:
        eng = pathtracer.Engine(ctx, 1 << 14)
        handles = []
        for k in range(9):
            desc = descs[k % 3]
            scene = pathtracer.upload_scene(ctx, desc)
            handles.append(scene.h.value)
            r = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
            eng.render([r], [4], use_graph=True)
            alone = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
            alone.rasterize_scene(4)
            assert np.allclose(r.film(), alone.film(), rtol=1e-5, atol=1e-7), k
            r.close()
            alone.close()
            scene.close()
        eng.close()
    assert len(set(handles)) < len(handles)   # an address came back
