"""A progress callback cuts a small request short.

The image's pool holds eight paths a pixel (65,536 for 8,192 pixels); a request
of 60 samples fits a larger pool whole, which a job with a callback must not get:
samples already given out run to their end.
"""
import numpy as np
import pytest

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu

SPP = 60


@pytest.mark.parametrize("before", [0, SPP])
def test_callback_stops_a_small_request(before):
    desc = scenes.cornell_box(width=128, height=64)
    with raycaster.Context(0) as ctx:
        scene = pathtracer.upload_scene(ctx, desc)
        r = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
        if before:
            r.rasterize_scene(before)   # leaves the larger pool behind
        r.set_progress(lambda done, total: False)
        assert r.rasterize_scene(SPP) is False
        spp = r.stats()["spp"]
        assert before < spp < before + SPP // 2
        whole = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
        whole.rasterize_scene(spp)
        assert np.allclose(r.film(), whole.film(), rtol=1e-5, atol=1e-7)
        r.set_progress(None)
        assert r.rasterize_scene(8) and r.stats()["spp"] == spp + 8
        seen = []
        r.set_progress(lambda done, total: seen.append((done, total)) or True)
        assert r.rasterize_scene(SPP)
        assert seen[0][0] < SPP and seen[-1] == (SPP, SPP)
        for x in (r, whole):
            x.close()
        scene.close()
