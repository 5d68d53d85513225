"""Casts from a warp's shared pools on both sides of the sizes where the
ray-per-lane caster takes over: 16,384 rays, 32,768 from 2^18 triangles up,
65,536 from 2^20; and bounce queues that start below that size, at it and above."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(5, 16384), (7, 32768), (8, 65536)], ids=["20K", "328K", "1.31M"])
def scene(rt, ctx, request):
    level, limit = request.param
    sc = ctx.upload_scene(rt.gen_icosphere(4, level), rt.gen_cornell(1, 0)[1])
    yield sc, limit
    sc.release()


def cast(ctx, sc, rays, flags, **tuning):
    import torch
    old = {k: ctx.get_tuning(k) for k in tuning}
    for k, v in tuning.items():
        ctx.set_tuning(k, v)
    try:
        hits = torch.full((len(rays), 4), 7.0, device="cuda")
        torch.cuda.synchronize()
        sc.trace(rays, len(rays), hits, flags)
        ctx.synchronize()
        return hits.cpu().numpy().view(np.uint32)
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)


@pytest.mark.parametrize("past", [-1, 0, 1])
def test_casts_around_the_limit_equal_ray_per_lane(rt, ctx, scene, past):
    import torch
    sc, limit = scene
    rays = rt.gen_random_rays(limit + past, limit + past)
    rays[::5, 7] = 1.2  # short rays
    rays[::7, 3] = 0.8
    rays = torch.from_numpy(rays).cuda()
    for flags in (0, rt.HIT_FP32):
        pooled = cast(ctx, sc, rays, flags)
        assert np.array_equal(pooled, cast(ctx, sc, rays, flags, **{"trace.packet_min_rays": 0, "trace.packet": 0}))


@pytest.mark.parametrize("width,height,spp", [(64, 64, 2), (128, 64, 2), (136, 60, 2), (182, 90, 1), (64, 64, 5), (256, 256, 1)])
def test_bounce_queues_around_the_limit(rt, ctx, width, height, spp):
    # 8,160 to 65,536 paths; a closed box keeps most of them through every bounce.
    import torch
    tris, mats, _ = rt.gen_cornell(8, 1500)
    sc = ctx.upload_scene(tris, mats)
    try:
        sc.set_camera(rt.camera_look_at([0, 0, -14], [0, 0, 0], [0, 1, 0], 40.0, width, height))
        out = []
        for mode in (0, 1):
            ctx.set_tuning("render.mode", mode)
            img = torch.zeros((height, width, 4), device="cuda")
            torch.cuda.synchronize()
            sc.render(img, width, height, spp=spp, max_bounces=8)
            ctx.synchronize()
            out.append(img)
        assert torch.equal(out[0], out[1])
    finally:
        ctx.set_tuning("render.mode", 2)
        sc.release()
