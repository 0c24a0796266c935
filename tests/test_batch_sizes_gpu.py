"""Ray casts of every batch size the feed treats apart.

Up to 32 rays per resident warp each warp gets an equal share, beyond that
warps take runs of 32 to 128 rays from a counter, and the last few rays of a
warp may be finished by all its lanes.  Sizes at the edges of these ranges on
a 148-SM device (4,736 resident warps at 8 blocks of 128 threads), on a soup
and on a tree deeper than the shared-memory stack.  The largest batch is held
to the oracle on a sample; every other batch gives the same answers bit by bit.
"""
import numpy as np
import pytest

import oracle
from rise_b200 import raycaster, scenes

from parity import any_report, closest_report

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 8, 9, 31, 33, 4735, 4737, 37888, 37889, 42000, 151552, 151553, 160000, 606208, 606209)
SAMPLE = 20_000


def soup():
    n = max(SIZES)
    return scenes.soup_triangles(20_000, seed=5), scenes.sphere_rays(n, 5), scenes.sphere_rays(n, 6, shadow=True)


def deep():
    tri = scenes.nested_clusters()
    return tri, scenes.cluster_rays(tri, max(SIZES), 5), scenes.cluster_rays(tri, max(SIZES), 6, shadow=True)


@pytest.mark.parametrize("layout", ["f32", "q8", "f16", "w8"])
@pytest.mark.parametrize("make", [soup, deep])
def test_batch_sizes_agree_and_match_the_oracle(make, layout):
    tri, rays, srays = make()
    with raycaster.Context(0) as ctx:
        s = raycaster.Scene(ctx)
        s.add_triangles(tri)
        s.commit(layout)
        rc = raycaster.RayCaster(s)
        hits, occ = rc.cast_rays(rays), rc.cast_shadow_rays(srays)
        ob = oracle.BVH(tri, "port")
        ids, t = ob.closest(rays[-SAMPLE:])
        rep = closest_report(tri, rays[-SAMPLE:], hits[-SAMPLE:], ids, t)
        assert rep["bad"] == [] and rep["t_over"] == 0, rep
        arep = any_report(tri, srays[-SAMPLE:], occ[-SAMPLE:], ob.any(srays[-SAMPLE:]))
        assert arep["bad"] == [], arep
        for n in SIZES:
            assert rc.cast_rays(rays[-n:]).tobytes() == hits[-n:].tobytes(), n
            assert rc.cast_shadow_rays(srays[-n:]).tobytes() == occ[-n:].tobytes(), n
        s.close()


def test_rays_with_nothing_to_hit():
    """NaN directions and empty ranges miss in every batch size."""
    tri = scenes.soup_triangles(2_000, seed=3)
    bad = scenes.sphere_rays(64, seed=3)
    bad[0::3, 4:7] = np.nan
    bad[1::3, 7] = 0.0
    bad[2::3, 3], bad[2::3, 7] = 5.0, 4.0
    with raycaster.Context(0) as ctx:
        s = raycaster.Scene(ctx)
        s.add_triangles(tri)
        s.commit("f16")
        rc = raycaster.RayCaster(s)
        for n in (1, 4, 64, 6400):
            rays = np.tile(bad, (100, 1))[:n]
            assert (rc.cast_rays(rays)["prim"] == -1).all()
            assert not rc.cast_shadow_rays(rays).any()
        s.close()
