"""Jobs whose engine is destroyed while their request is in flight.

A short request is withdrawn, as if it had not been made; one whose samples are
already in the job's sums ends at the pixel samples started.  Either way the job's
film is a whole number of samples, read or not, and rendering goes on from there.
"""
import dataclasses

import numpy as np
import pytest

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.allclose(a, b, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("read", [False, True])
@pytest.mark.parametrize("spp,steps,settings", [
    (16, 2, {}), (16, 2, {"filter": 1}), (48, 1, {"filter": 1, "sampler": 2}), (16, 0, {"filter": 1}),
    (128, 2, {}), (128, 2, {"filter": 1}), (128, 0, {}),
    (40, 2, {"adaptive_max_spp": 96, "adaptive_threshold": 0.2}),
])
def test_job_is_whole_after_its_engine_goes(spp, steps, settings, read):
    desc = scenes.cornell_box(width=48, height=40)
    st = dataclasses.replace(desc.settings, **settings)
    with raycaster.Context(0) as ctx:
        scene = pathtracer.upload_scene(ctx, desc)

        def job():
            return pathtracer.SpectralRasterizer(ctx, desc, scene=scene, settings=st)

        cut, whole = job(), job()
        eng = pathtracer.Engine(ctx, 1 << 13)
        cut.rasterize_scene(4)
        whole.rasterize_scene(4)
        eng.submit(cut, spp)
        for _ in range(steps):
            eng.step(2, use_graph=False)
        assert not steps or 0 < eng.progress(cut)[0] < eng.progress(cut)[1]
        eng.close()
        k = cut.stats()["spp"] - 4
        if steps and (spp >= 64 or "adaptive_max_spp" in settings):
            assert 0 < k < spp
            whole.rasterize_scene(k)
        else:
            assert k == 0
        if read:
            assert same(cut.film(), whole.film())
        cut.rasterize_scene(12)
        whole.rasterize_scene(12)
        assert same(cut.film(), whole.film())
        assert np.array_equal(cut.sample_counts(), whole.sample_counts())
        for x in (cut, whole):
            x.close()
        scene.close()


def test_scene_gone_first():
    """Nothing runs for a scene that is gone; the job says that it lost samples."""
    desc = scenes.cornell_box(width=48, height=40)
    with raycaster.Context(0) as ctx:
        scene = pathtracer.upload_scene(ctx, desc)
        other = pathtracer.upload_scene(ctx, desc)
        r = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
        late = pathtracer.SpectralRasterizer(ctx, desc, scene=other)
        eng = pathtracer.Engine(ctx, 1 << 13)
        eng.submit(r, 128)
        eng.submit(late, 16)
        eng.step(2, use_graph=False)
        other.close()
        eng.close()
        for call in (r.film, r.rgb, r.sample_counts, lambda: r.rasterize_scene(1)):
            with pytest.raises(Exception) as e:
                call()
            assert "E_DEVICE" in str(e.value)
        r.close()
        scene.close()
