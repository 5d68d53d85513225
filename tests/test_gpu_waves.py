"""The wavefront's sample waves against the megakernel, bit for bit: partial
8 x 4 tiles, calls cut into several waves, every bounce count at which the
launch sequence changes, and each caster of the bounce rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def render(rt, ctx, sc, width, height, start, mode, **kw):
    import torch
    ctx.set_tuning("render.mode", mode)
    try:
        img = torch.from_numpy(start).cuda()
        torch.cuda.synchronize()
        ctx.segments(reset=True)
        sc.render(img, width, height, **kw)
        ctx.synchronize()
        return img.cpu().numpy(), ctx.segments()
    finally:
        ctx.set_tuning("render.mode", 2)


@pytest.mark.parametrize("width,height,spp,bounces", [
    (1, 1, 5, 8), (7, 3, 3, 8), (33, 5, 2, 1), (31, 18, 4, 0), (64, 48, 1, 2), (100, 37, 7, 3),
    (600, 601, 5, 4),    # two samples a wave and a last wave of one
    (1024, 1026, 2, 3),  # more tile positions than a wave of paths
])
def test_waves_equal_the_megakernel(rt, ctx, width, height, spp, bounces):
    tris, mats, sph = rt.gen_cornell(5, 1500, 3)
    sc = ctx.upload_scene(tris, mats, spheres=sph)
    try:
        sc.set_camera(rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, width, height))
        start = np.random.RandomState(width).rand(height, width, 4).astype(np.float32)
        for kw in (dict(sample_index=0), dict(sample_index=3, flags=rt.COMPAT_UNORM8)):
            want, seg = render(rt, ctx, sc, width, height, start, 0, spp=spp, max_bounces=bounces, **kw)
            got, seg1 = render(rt, ctx, sc, width, height, start, 1, spp=spp, max_bounces=bounces, **kw)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and seg == seg1
    finally:
        sc.release()


@pytest.mark.parametrize("tuning", [{"render.sort": 1}, {"trace.wide": 0}, {"trace.wide": 0, "render.sort": 1}])
def test_waves_on_every_caster(rt, ctx, tuning):
    tris, mats, _ = rt.gen_cornell(6, 2500)
    sc = ctx.upload_scene(tris, mats)
    old = {k: ctx.get_tuning(k) for k in tuning}
    try:
        sc.set_camera(rt.camera_look_at([0, 0, -14], [0, 0, 0], [0, 1, 0], 40.0, 150, 90))
        start = np.zeros((90, 150, 4), np.float32)
        want, seg = render(rt, ctx, sc, 150, 90, start, 0, spp=3, max_bounces=6)
        for k, v in tuning.items():
            ctx.set_tuning(k, v)
        got, seg1 = render(rt, ctx, sc, 150, 90, start, 1, spp=3, max_bounces=6)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and seg == seg1
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)
        sc.release()
