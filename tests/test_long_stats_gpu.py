"""Ray statistics of a kept engine go on past 2^32 rays."""
import pytest

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu


def test_shadow_ray_count_passes_32_bits():
    desc = scenes.cornell_box(width=256, height=256)
    with raycaster.Context(0) as ctx:
        r = pathtracer.SpectralRasterizer(ctx, desc)
        counts = []
        while not counts or counts[-1][0] < 2 ** 32 + 2 ** 30:
            r.rasterize_scene(512)
            st = r.stats()
            assert len(counts) < 64
            counts.append((st["shadow_rays"], st["segments"]))
        for k in range(2):
            # Every request of 512 samples a pixel casts about as many rays.
            steps = [b[k] - a[k] for a, b in zip(counts, counts[1:])]
            assert counts[0][k] > 0 and all(abs(x - counts[0][k]) < 0.01 * counts[0][k] for x in steps)
        r.close()
