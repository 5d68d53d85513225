"""Casts and small renders from a warp's shared pools (pool.cu, paths.cu)
against the ray-per-lane and megakernel forms, bit for bit: batch and image
sizes around the changes of rays per warp, scenes whose rays fill the pools,
one-triangle scenes, and device-sized queues on either side of the limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cast(rt, ctx, sc, rays, direct, flags=0):
    import torch
    old = ctx.get_tuning("trace.packet_min_rays")
    ctx.set_tuning("trace.packet_min_rays", 1 << 30 if direct else 0)
    ctx.set_tuning("trace.packet", 1 if direct else 0)  # 0: every ray on the ray-per-lane caster
    try:
        d_rays = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
        d_hits = torch.full((len(rays), 4), 7.0, device="cuda")
        torch.cuda.synchronize()
        sc.trace(d_rays, len(rays), d_hits, flags)
        ctx.synchronize()
        return d_hits.cpu().numpy().view(np.uint32)
    finally:
        ctx.set_tuning("trace.packet_min_rays", old)
        ctx.set_tuning("trace.packet", 1)


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 100, 8191, 8192, 8193, 32768, 32769])
def test_pool_casts_equal_ray_per_lane(rt, ctx, n):
    sc = ctx.upload_scene(rt.gen_icosphere(4, 5), rt.gen_cornell(1, 0)[1])
    try:
        rays = rt.gen_random_rays(n, n)
        rays[::5, 7] = 1.2  # short rays
        rays[::7, 3] = 0.8
        for flags in (0, rt.HIT_FP32):
            assert np.array_equal(cast(rt, ctx, sc, rays, True, flags), cast(rt, ctx, sc, rays, False, flags))
    finally:
        sc.release()


@pytest.mark.parametrize("case", ["one", "two", "coincident", "overlapping", "flat"])
def test_degenerate_scenes(rt, ctx, case):
    # Coincident and widely overlapping triangles enter every child of every
    # node: the pools run to their limits.
    tris, mats, _ = rt.gen_cornell(3, 3000)
    tris = tris[12:]
    if case in ("one", "two"):
        tris = tris[: 1 if case == "one" else 2]
    elif case == "coincident":
        tris = np.tile(tris[:1], (3000, 1))
    elif case == "overlapping":
        for v in (0, 4, 8):
            tris[:, v:v + 3] = np.random.RandomState(v).uniform(-4, 4, (len(tris), 3))
    else:
        for v in (0, 4, 8):
            tris[:, v + 1] = 0.5
    sc = ctx.upload_scene(tris, mats)
    try:
        rays = rt.gen_random_rays(11, 3000, -5, 5)
        rays[::3, 5] = 0.0  # and axis-parallel ones
        rays[::9, 4] = 0.0
        assert np.array_equal(cast(rt, ctx, sc, rays, True), cast(rt, ctx, sc, rays, False))
    finally:
        sc.release()


@pytest.mark.parametrize("width,height", [(1, 1), (9, 5), (64, 32), (90, 91), (128, 129), (256, 255), (256, 256)])
def test_small_renders_equal_the_megakernel(rt, ctx, width, height):
    import torch
    tris, mats, sph = rt.gen_cornell(8, 1500, 3)
    sc = ctx.upload_scene(tris, mats, spheres=sph)
    try:
        sc.set_camera(rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, width, height))
        for kw in (dict(max_bounces=8), dict(max_bounces=1, sample_index=4), dict(max_bounces=3, flags=rt.SHADE_SIMPLE),
                   dict(max_bounces=0), dict(max_bounces=5, sample_index=2, flags=rt.COMPAT_UNORM8)):
            out = []
            for mode in (0, 2, 3):
                ctx.set_tuning("render.mode", mode)
                img = torch.full((height, width, 4), 0.25, device="cuda")
                torch.cuda.synchronize()
                ctx.segments(reset=True)
                sc.render(img, width, height, spp=1, **kw)
                ctx.synchronize()
                out.append((img.cpu().numpy().view(np.uint32), ctx.segments()))
            assert all(np.array_equal(o[0], out[0][0]) and o[1] == out[0][1] for o in out[1:]), kw
    finally:
        ctx.set_tuning("render.mode", 2)
        sc.release()


@pytest.mark.parametrize("side", [100, 182, 200])
def test_bounce_queues_on_either_side_of_the_limit(rt, ctx, side):
    # 10,000 to 40,000 paths a sample: the queues of a call start above or
    # below 32,768 and shrink through it.
    import torch
    tris, mats, _ = rt.gen_cornell(8, 1500)
    sc = ctx.upload_scene(tris, mats)
    try:
        sc.set_camera(rt.camera_look_at([0, 0, -14], [0, 0, 0], [0, 1, 0], 40.0, side, side))
        out = []
        for mode in (0, 1):
            ctx.set_tuning("render.mode", mode)
            img = torch.zeros((side, side, 4), device="cuda")
            torch.cuda.synchronize()
            sc.render(img, side, side, spp=2, max_bounces=8)
            ctx.synchronize()
            out.append(img.cpu().numpy().view(np.uint32))
        assert np.array_equal(out[0], out[1])
    finally:
        ctx.set_tuning("render.mode", 2)
        sc.release()
