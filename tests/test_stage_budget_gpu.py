"""Casts of host arrays stage no more than the whole batch."""
import pytest

from rise_b200 import raycaster, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 131_072, 131_073, 200_001, 262_144])
def test_batch_fits_a_budget_of_its_own_size(n):
    tri, rays = scenes.soup_triangles(2_000, seed=3), scenes.sphere_rays(n, 3)
    answers, held = [], 0
    for shadow in (False, True):
        for tight in (False, True):
            with raycaster.Context(0, held + n * (33 if shadow else 48) if tight else 0) as ctx:
                s = raycaster.Scene(ctx)
                s.add_triangles(tri)
                s.commit("f32")
                held = ctx.bytes_in_use()
                rc = raycaster.RayCaster(s)
                answers.append((rc.cast_shadow_rays if shadow else rc.cast_rays)(rays).tobytes())
                s.close()
    assert answers[0] == answers[1] and answers[2] == answers[3]
