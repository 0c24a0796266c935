"""Memory that closed jobs and engines leave to the next ones can be given back."""
import numpy as np
import pytest
import torch

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu


def test_trim_frees_what_closed_jobs_and_engines_left():
    desc = scenes.cornell_box(width=128, height=96)
    with raycaster.Context(0) as ctx:
        scene = pathtracer.upload_scene(ctx, desc)

        def image():
            r = pathtracer.SpectralRasterizer(ctx, desc, scene=scene)
            r.rasterize_scene(48)
            img = r.film()
            r.close()
            return img

        first = image()
        pathtracer.Engine(ctx, 1 << 20).close()
        held = ctx.bytes_in_use()
        free = torch.cuda.mem_get_info()[0]
        ctx.trim()
        assert torch.cuda.mem_get_info()[0] - free > 400 << 20   # 256 bytes and more a path, 1.5 M paths
        assert ctx.bytes_in_use() == held
        assert np.allclose(image(), first, rtol=1e-5, atol=1e-7)
        ctx.trim()
        ctx.trim()
        scene.close()
        assert ctx.bytes_in_use() == 0
