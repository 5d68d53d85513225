"""Renders of small images in captured graphs and on several streams: every
image bit for bit, whatever else is under way, and no memory of a graph's own
where the call was one launch."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(rt, ctx, soup=1500, side=128):
    tris, mats, _ = rt.gen_cornell(8, soup)
    sc = ctx.upload_scene(tris, mats)
    sc.set_camera(rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, side, side))
    return sc


def captured(sc, image, width, height, **kw):
    """A graph of one render call, kept so that its nodes can be read."""
    import torch
    g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        sc.render(image, width, height, stream=s.cuda_stream, **kw)
    return g


def node_types(graph):
    """The kinds of the graph's nodes (CUgraphNodeType)."""
    drv = ctypes.CDLL("libcuda.so.1")
    g, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert drv.cuGraphGetNodes(g, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert drv.cuGraphGetNodes(g, nodes, ctypes.byref(n)) == 0
    out = []
    for node in nodes:
        t = ctypes.c_int(-1)
        assert drv.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(t)) == 0
        out.append(t.value)
    return out


KERNEL, MEM_ALLOC, MEM_FREE = 0, 10, 11


@pytest.mark.parametrize("spp", [1, 3])
@pytest.mark.parametrize("side", [64, 256, 362, 363, 400, 511])
def test_captured_renders_are_one_launch(rt, ctx, side, spp):
    import torch
    sc = scene(rt, ctx, side=side)
    try:
        image, want = torch.zeros((side, side, 4), device="cuda"), torch.zeros((side, side, 4), device="cuda")
        g = captured(sc, image, side, side, spp=spp, max_bounces=5)
        types = node_types(g)
        assert MEM_ALLOC not in types and MEM_FREE not in types and types.count(KERNEL) == 1
        g.instantiate()
        g.replay()
        torch.cuda.synchronize()
        sc.render(want, side, side, spp, 5)
        ctx.synchronize()
        assert torch.equal(image, want)
    finally:
        sc.release()


def test_replays_and_live_calls_keep_their_own_counters(rt, ctx):
    # A captured render at sample 3 replayed on one stream beside more calls
    # than the context has counter words on another.
    import torch
    sc = scene(rt, ctx)
    try:
        start = torch.from_numpy(np.random.RandomState(1).rand(128, 128, 4).astype(np.float32)).cuda()
        ray = torch.from_numpy(rt.gen_random_rays(2, 1000, -4, 4)).cuda()
        want, want64, hits = start.clone(), torch.zeros((64, 64, 4), device="cuda"), torch.zeros((1000, 4), device="cuda")
        torch.cuda.synchronize()
        sc.render(want, 128, 128, 1, 8, sample_index=3)
        sc.render(want64, 64, 64, 1, 8)
        sc.trace(ray, 1000, hits)
        ctx.synchronize()
        image = start.clone()
        g = captured(sc, image, 128, 128, spp=1, max_bounces=8, sample_index=3)
        g.instantiate()
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        live = [(torch.zeros_like(want64), torch.full_like(hits, 7.0)) for _ in range(60)]
        copies = [torch.empty_like(image) for _ in range(40)]
        torch.cuda.synchronize()
        k = 0
        for i in range(40):
            with torch.cuda.stream(a):
                image.copy_(start)
                g.replay()
                copies[i].copy_(image)
            for _ in range(60):
                img, hit = live[k % 60]
                sc.trace(ray, 1000, hit, 0, b.cuda_stream)
                if k % 4 == 0:
                    sc.render(img, 64, 64, 1, 8, stream=b.cuda_stream)
                k += 1
        torch.cuda.synchronize()
        assert all(torch.equal(c, want) for c in copies)
        assert all(torch.equal(h.view(torch.int32), hits.view(torch.int32)) for _, h in live)
        assert all(torch.equal(i, want64) for i, _ in live[::4])
    finally:
        sc.release()


def test_a_stream_held_back_keeps_its_counter(rt, ctx):
    import torch
    sc = scene(rt, ctx)
    try:
        big = torch.zeros((1500, 1500, 4), device="cuda")
        images = [torch.zeros((96, 96, 4), device="cuda") for _ in range(8)]
        other, want = torch.zeros((96, 96, 4), device="cuda"), torch.zeros((96, 96, 4), device="cuda")
        torch.cuda.synchronize()
        for s in range(2):
            sc.render(want, 96, 96, 1, 8, sample_index=s)
        ctx.synchronize()
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        for img in images:  # each waits for a long call, more than 1,024 on the other stream go past
            sc.render(big, 1500, 1500, 2, 8, stream=a.cuda_stream)
            for s in range(2):
                sc.render(img, 96, 96, 1, 8, sample_index=s, stream=a.cuda_stream)
        for _ in range(1100):
            sc.render(other, 16, 16, 1, 1, stream=b.cuda_stream)
        torch.cuda.synchronize()
        assert all(torch.equal(i, want) for i in images)
    finally:
        sc.release()
