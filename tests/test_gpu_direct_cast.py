"""Batches that go straight to the 8-wide caster (trace.packet_min_rays)
against the sort and packet path, bit for bit: batch sizes around a warp, a
block and the sort's threshold, the gate that tells camera batches from
random ones, and the host entry point's chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(rt, ctx):
    sc = ctx.upload_scene(rt.gen_icosphere(8, 5), rt.gen_cornell(1, 0)[1])
    yield sc
    sc.release()


def rays_of(rt, kind, n):
    side = int(np.ceil(np.sqrt(n)))
    cams = [rt.gen_camera_rays(rt.camera_look_at(eye, [0, 0, 0], [0, 1, 0], 40.0, side, side), side, side)[:n]
            for eye in ([0, 0, -3], [0.5, 1, -2.5])]
    if kind == "camera":
        return cams[0]
    if kind == "two cameras in turn":
        return np.where((np.arange(n) % 2 == 0)[:, None], cams[0], cams[1]).astype(np.float32)
    if kind == "half camera":
        return np.concatenate([cams[0][:n // 2], rt.gen_random_rays(9, n - n // 2)])
    return rt.gen_random_rays(9, n)


def cast(rt, ctx, sc, rays, min_rays, host=False, flags=0):
    import torch
    old = ctx.get_tuning("trace.packet_min_rays")
    ctx.set_tuning("trace.packet_min_rays", min_rays)
    try:
        if host:
            return sc.trace_host(rays)
        d_rays = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
        d_hits = torch.full((len(rays), 4), 7.0, device="cuda")
        torch.cuda.synchronize()
        sc.trace(d_rays, len(rays), d_hits, flags)
        ctx.synchronize()
        return d_hits.cpu().numpy()
    finally:
        ctx.set_tuning("trace.packet_min_rays", old)


@pytest.mark.parametrize("kind", ["camera", "random", "half camera", "two cameras in turn"])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 5000, 65535, 65536, 200003])
def test_direct_equals_sorted_packets(rt, ctx, scene, n, kind):
    rays = rays_of(rt, kind, n)
    for flags in (0, rt.HIT_FP32):
        packets = cast(rt, ctx, scene, rays, 0, flags=flags)  # gated from 65,536 rays up
        direct = cast(rt, ctx, scene, rays, 1 << 30, flags=flags)
        assert np.array_equal(packets.view(np.uint32), direct.view(np.uint32))


@pytest.mark.parametrize("kind", ["camera", "random"])
def test_host_chunks_equal_device_casts(rt, ctx, scene, kind):
    rays = rays_of(rt, kind, 150001)
    want = cast(rt, ctx, scene, rays, 1 << 30)
    old = ctx.get_tuning("trace.host_chunk")
    try:
        for chunk in (65536, old):
            ctx.set_tuning("trace.host_chunk", chunk)
            for min_rays in (0, 1 << 30):
                got = cast(rt, ctx, scene, rays, min_rays, host=True)
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    finally:
        ctx.set_tuning("trace.host_chunk", old)
