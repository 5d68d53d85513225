"""Rays that start far from a mesh near the origin: within 400 units every tree
and every casting kernel gives the same hits, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 200000


def cast(rt, ctx, sc, rays, **tuning):
    import torch
    old = {k: ctx.get_tuning(k) for k in tuning}
    for k, v in tuning.items():
        ctx.set_tuning(k, v)
    try:
        hits = torch.zeros((len(rays), 4), device="cuda")
        torch.cuda.synchronize()
        sc.trace(rays, len(rays), hits)
        ctx.synchronize()
        return hits.cpu().numpy().view(np.uint32)
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)


def upload(rt, ctx, tris, mats, **tuning):
    old = {k: ctx.get_tuning(k) for k in tuning}
    for k, v in tuning.items():
        ctx.set_tuning(k, v)
    try:
        return ctx.upload_scene(tris, mats)
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)


@pytest.mark.parametrize("distance", [100, 250, 400])
@pytest.mark.parametrize("mesh", ["icosphere", "cornell"])
def test_distant_rays_hit_the_same_on_every_route(rt, ctx, mesh, distance):
    import torch
    mats = rt.gen_cornell(1, 0)[1]
    tris = rt.gen_icosphere(12, 5) if mesh == "icosphere" else rt.gen_cornell(12, 5000)[0]
    rays = rt.gen_random_rays(7, N) if mesh == "icosphere" else rt.gen_random_rays(7, N, -5, 5)
    rays[:, 0:3] -= np.float32(distance) * rays[:, 4:7]
    cam = rt.camera_look_at([0.1 * distance, 0.2 * distance, -0.97 * distance], [0, 0, 0], [0, 1, 0], 1.5, 300, 200)
    d_rays = torch.from_numpy(np.concatenate([rays, rt.gen_camera_rays(cam, 300, 200)])).cuda()
    scenes = [upload(rt, ctx, tris, mats, **t) for t in
              ({"bvh.cast_tree": 0}, {"bvh.cast_tree": 1}, {"bvh.builder": 1}, {"bvh.builder": 2})]
    try:
        want = cast(rt, ctx, scenes[0], d_rays, **{"trace.wide": 0})
        assert (want[:, 0] != 0xffffffff).sum() > N // 4
        for sc in scenes:
            for tuning in ({}, {"trace.packet_min_rays": 0}, {"trace.wide": 0}):
                assert np.array_equal(cast(rt, ctx, sc, d_rays, **tuning), want), tuning
        pooled = d_rays[:16000].contiguous()
        for sc in scenes:
            assert np.array_equal(cast(rt, ctx, sc, pooled), want[:16000])
    finally:
        for sc in scenes:
            sc.release()
