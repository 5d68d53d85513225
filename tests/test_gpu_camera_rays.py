"""Wavefront renders whose camera rays are cast as rays of their own (many
triangles a pixel) against the megakernel, bit for bit: ragged images on either
side of the rule, image and batch forms, one sample and several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (33, 17), (100, 61), (160, 169), (161, 170), (257, 200)])
def test_own_camera_rays_keep_the_image(rt, ctx, w, h):
    import torch
    mats = rt.gen_cornell(1, 0)[1]
    sc = ctx.upload_scene(rt.gen_icosphere(8, 6), mats)  # 81,920 triangles: own rays up to 27,306 tile positions
    cam = rt.camera_look_at([0, 0.3, -3], [0, 0, 0], [0, 1, 0], 45.0, w, h)
    sc.set_camera(cam)
    old = ctx.get_tuning("render.mode")
    images = []
    try:
        for mode in (0, 1):
            ctx.set_tuning("render.mode", mode)
            for spp in (1, 3):
                img = torch.zeros((h, w, 4), device="cuda")
                torch.cuda.synchronize()
                sc.render(img, w, h, spp, 4)
                ctx.synchronize()
                images.append(img.cpu().numpy())
    finally:
        ctx.set_tuning("render.mode", old)
    batched = torch.zeros((h, w, 4), device="cuda")
    torch.cuda.synchronize()
    ctx.render_batch([rt.make_job(sc, cam, batched, w, h, 3, 4)])
    ctx.synchronize()
    sc.release()
    for a, c in zip(images[:2], images[2:]):
        assert np.array_equal(a.view(np.uint32), c.view(np.uint32))
    assert np.array_equal(batched.cpu().numpy().view(np.uint32), images[1].view(np.uint32))
