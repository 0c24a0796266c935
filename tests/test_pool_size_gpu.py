"""The path pool of a job's own engine: its size changes no image.

A small image gets a pool as large as its request; a later, larger request
enlarges it, and one that folds its film step by step (64 samples per pixel on)
or a context with a memory budget keeps the small one.
"""
import dataclasses

import numpy as np
import pytest

from rise_b200 import pathtracer, raycaster, scenes

pytestmark = pytest.mark.gpu


def render(ctx, desc, spp, **settings):
    r = pathtracer.SpectralRasterizer(ctx, desc, settings=dataclasses.replace(desc.settings, **settings))
    used = []
    for n in spp:
        r.rasterize_scene(n)
        used.append(ctx.bytes_in_use())
    img = r.film()
    r.close()
    return img.astype(np.float64), used


def same(a, b):
    # Only the order of FP32 film additions differs.
    return np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


@pytest.mark.parametrize("size", [(1, 1), (33, 7), (128, 96)])
def test_pool_size_does_not_change_the_image(size):
    desc = scenes.cornell_box(width=size[0], height=size[1])
    with raycaster.Context(0) as ctx:
        few, _ = render(ctx, desc, [48, 64], max_paths=4096)
        once, _ = render(ctx, desc, [112])
        grown, used = render(ctx, desc, [1, 47, 64])
        assert same(once, few) and same(grown, few)
        assert used[1] >= used[0] == used[2]
        assert ctx.bytes_in_use() == 0


def test_budget_keeps_the_small_pool():
    desc = scenes.cornell_box(width=128, height=96)
    with raycaster.Context(0) as ctx:
        _, free = render(ctx, desc, [48])
    with raycaster.Context(0, 256 << 20) as ctx:
        _, tight = render(ctx, desc, [48])
    assert tight[0] < 128 << 20 < free[0]
