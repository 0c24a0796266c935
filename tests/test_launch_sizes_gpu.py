"""One launch of every size the feed and the choice of kernels treat apart.

Rays and answers stay on the device, so that a batch is one launch (casts of host
arrays are cut into pieces).  The sizes lie at the edges of what one device
does: an equal share for each warp up to 32 rays a resident warp, runs from a
counter beyond, and from 4,096 rays per SM on the kernels whose warps do not join
forces for their last rays.  On the soup the largest batch is held to the oracle
on a sample (the deep tree's coordinates of 1e3 put FP32 edges outside the band
that the comparison excludes); the others give its answers bit by bit, and so do
host arrays.
"""
import numpy as np
import pytest
import torch

import oracle
from rise_b200 import raycaster, scenes

from parity import any_report, closest_report

pytestmark = pytest.mark.gpu

SAMPLE = 20_000


def sizes():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    share, joint = 32 * 32 * sms, 4096 * sms   # 32 resident warps an SM
    return (1, 33, share - 1, share, share + 1, 8 * 32 * 32 * sms // 2 + 3, joint - 1, joint, joint + 1, 2 * joint + 77,
            3 * joint + 5)


def soup(n):
    return scenes.soup_triangles(20_000, seed=5), scenes.sphere_rays(n, 5), scenes.sphere_rays(n, 6, shadow=True)


def deep(n):
    tri = scenes.nested_clusters()
    return tri, scenes.cluster_rays(tri, n, 5), scenes.cluster_rays(tri, n, 6, shadow=True)


@pytest.mark.parametrize("layout", ["f32", "q8", "f16", "w8"])
@pytest.mark.parametrize("make", [soup, deep])
def test_one_launch_agrees_and_matches_the_oracle(make, layout):
    top = max(sizes())
    tri, rays, srays = make(top)
    d_rays, d_srays = torch.from_numpy(rays).cuda(), torch.from_numpy(srays).cuda()
    stream = torch.cuda.current_stream().cuda_stream
    with raycaster.Context(0) as ctx:
        s = raycaster.Scene(ctx)
        s.add_triangles(tri)
        s.commit(layout)
        rc = raycaster.RayCaster(s)

        def cast(n):
            hits = torch.empty(n, 4, device="cuda")
            occ = torch.empty(n, dtype=torch.uint8, device="cuda")
            rc.cast_rays_device(d_rays[top - n:].data_ptr(), hits.data_ptr(), n, stream)
            rc.cast_shadow_rays_device(d_srays[top - n:].data_ptr(), occ.data_ptr(), n, stream)
            return hits.view(torch.int32), occ

        hits, occ = cast(top)
        last = hits[-SAMPLE:].cpu().numpy().view(raycaster.HIT_DTYPE)[:, 0]
        last_occ = occ[-SAMPLE:].cpu().numpy()
        assert rc.cast_rays(rays[-SAMPLE:]).tobytes() == last.tobytes()
        assert rc.cast_shadow_rays(srays[-SAMPLE:]).tobytes() == last_occ.tobytes()
        if make is soup:
            ob = oracle.BVH(tri, "port")
            ids, t = ob.closest(rays[-SAMPLE:])
            rep = closest_report(tri, rays[-SAMPLE:], last, ids, t)
            assert rep["bad"] == [] and rep["t_over"] == 0, rep
            arep = any_report(tri, srays[-SAMPLE:], last_occ, ob.any(srays[-SAMPLE:]))
            assert arep["bad"] == [], arep
        for n in sizes():
            h, o = cast(n)
            assert torch.equal(h, hits[-n:]), n
            assert torch.equal(o, occ[-n:]), n
        s.close()
