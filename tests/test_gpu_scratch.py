"""The context's scratch pool: calls on several streams and from several
threads, with synchronisations between them, give the hits and trees of calls
made one after the other, and what the pool keeps is bounded and given back."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_and_streams_share_the_pool(rt, ctx):
    import torch
    tris, mats = rt.gen_icosphere(5, 5), rt.gen_cornell(1, 0)[1]
    sc = ctx.upload_scene(tris, mats)
    cam = rt.camera_look_at([0, 0, -3], [0, 0, 0], [0, 1, 0], 40.0, 1200, 1000)
    sc.set_camera(cam)
    rays = torch.from_numpy(rt.gen_camera_rays(cam, 1200, 1000)).cuda()  # sorted: takes scratch
    want = torch.zeros((len(rays), 4), device="cuda")
    image = torch.zeros((1000, 1200, 4), device="cuda")
    torch.cuda.synchronize()
    sc.trace(rays, len(rays), want)
    sc.render(image, 1200, 1000, 1, 4)
    ctx.synchronize()
    bad = []

    def work(i):
        st = torch.cuda.Stream()
        got = torch.zeros_like(want)
        img = torch.zeros_like(image)
        torch.cuda.synchronize()
        for k in range(4):
            sc.trace(rays, len(rays), got, 0, st.cuda_stream)
            sc.render(img, 1200, 1000, 1, 4, stream=st.cuda_stream)
            if k % 2 == i % 2:
                st.synchronize()
        st.synchronize()
        if not torch.equal(got.view(torch.int32), want.view(torch.int32)) or not torch.equal(img, image):
            bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    sc.release()
    assert not bad


def test_kept_scratch_is_bounded_and_given_back(rt):
    import torch
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    own = rt.Context(0)
    mats = rt.gen_cornell(1, 0)[1]
    for level in (8, 7):
        sc = own.upload_scene(rt.gen_icosphere(1, level), mats)
        sc.release()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= (1 << 30) + (256 << 20)
    own.close()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 256 << 20
