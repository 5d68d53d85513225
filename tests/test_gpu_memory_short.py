"""Calls that meet a shortage of device memory: what they refuse and return is
what they do with memory to spare."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def tune(ctx):
    """Sets tuning keys for one test."""
    old = {}

    def set_(**kw):
        for k, v in kw.items():
            key = k.replace("__", ".")
            old.setdefault(key, ctx.get_tuning(key))
            ctx.set_tuning(key, v)

    yield set_
    for k, v in old.items():
        ctx.set_tuning(k, v)


def soup(rt, n):
    tris, mats, _ = rt.gen_cornell(n, n)
    return np.ascontiguousarray(tris[12:]), mats


@pytest.mark.parametrize("n", [32768, 40003])
def test_a_check_that_runs_out_of_memory_leaves_the_hosts(rt, ctx, tune, n):
    tris, mats = soup(rt, n)
    light = int(np.flatnonzero(mats.view(np.uint32)[:, 0] == rt.MATERIAL_LIGHT)[0])
    tris.view(np.uint32)[::97, 11] = light
    tune(scene__test_stage_error=1)
    for word, value in ((0, np.nan), (10, np.inf)):
        bad = tris.copy()
        bad[n // 2, word] = value
        with pytest.raises(rt.RtError) as e:
            ctx.upload_scene(bad, mats)
        assert e.value.status == 5 and f"triangle {n // 2}: non-finite vertex" in str(e.value)
    bad = tris.copy()
    bad.view(np.uint32)[n - 1, 11] = 0x7fffffff
    with pytest.raises(rt.RtError) as e:
        ctx.upload_scene(bad, mats)
    assert e.value.status == 5 and f"triangle {n - 1}: material" in str(e.value)
    sc = ctx.upload_scene(tris, mats)
    try:
        want = rt.lights_from_materials(tris, mats)
        assert len(want) and np.array_equal(sc.lights().view(np.uint32), want.view(np.uint32))
    finally:
        sc.release()


@pytest.mark.parametrize("spp", [1, 3])
@pytest.mark.parametrize("side", [48, 256, 362, 363, 400, 511])
def test_renders_without_scratch_are_one_launch(rt, ctx, tune, side, spp):
    import torch
    tris, mats, _ = rt.gen_cornell(8, 1500)
    sc = ctx.upload_scene(tris, mats)
    try:
        sc.set_camera(rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, side, side))
        images = []
        for limit in (0, 1):
            tune(test__alloc_limit=limit)
            img = torch.zeros((side, side, 4), device="cuda")
            torch.cuda.synchronize()
            sc.render(img, side, side, spp, 5)
            ctx.synchronize()
            images.append(img)
        assert torch.equal(images[0], images[1])
        big = torch.zeros((512, 512, 4), device="cuda")
        with pytest.raises(rt.RtError):  # from 2^18 pixels the scratch is a condition
            sc.render(big, 512, 512, spp, 5)
    finally:
        tune(test__alloc_limit=0)
        sc.release()


def one_sample_limit(side):
    """Bytes that hold a sample's paths of a side x side image, not two samples'."""
    return 140 * side * side


def test_large_renders_take_a_sample_at_a_time(rt, ctx, tune):
    import torch
    tris, mats, _ = rt.gen_cornell(8, 1500)
    sc = ctx.upload_scene(tris, mats)
    try:
        sc.set_camera(rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, 512, 512))
        images = []
        for limit in (0, one_sample_limit(512)):
            tune(test__alloc_limit=limit)
            img = torch.zeros((512, 512, 4), device="cuda")
            torch.cuda.synchronize()
            sc.render(img, 512, 512, 4, 5)
            ctx.synchronize()
            images.append(img)
        assert torch.equal(images[0], images[1])
    finally:
        tune(test__alloc_limit=0)
        sc.release()


def test_batches_take_a_sample_at_a_time(rt, ctx, tune):
    import torch
    scenes = [ctx.upload_scene(*rt.gen_cornell(8 + i, 1500)[:2]) for i in range(3)]
    try:
        cam = rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, 128, 128)
        images = []
        for limit in (0, one_sample_limit(128)):
            tune(test__alloc_limit=limit)
            imgs = [torch.zeros((128, 128, 4), device="cuda") for _ in scenes]
            torch.cuda.synchronize()
            b = ctx.batch([rt.make_job(s, cam, i, 128, 128, 16, 4) for s, i in zip(scenes, imgs)])
            b.launch()
            ctx.synchronize()
            b.launch_graph()
            ctx.synchronize()
            b.destroy()
            images.append(imgs)
        assert all(torch.equal(a, b) for a, b in zip(*images))
        tune(test__alloc_limit=1000)
        with pytest.raises(rt.RtError):
            ctx.batch([rt.make_job(scenes[0], cam, images[0][0], 128, 128, 16, 4)])
    finally:
        tune(test__alloc_limit=0)
        for s in scenes:
            s.release()


def test_the_server_takes_a_sample_at_a_time(rt, ctx, tune):
    from rtgb import serve
    data = rt.gen_cornell(8, 300)
    cam = rt.camera_look_at([0.2, 0.1, -14], [0, 0, 0], [0, 1, 0], 40.0, 128, 128)
    images = []
    for limit in (0, one_sample_limit(128)):
        tune(test__alloc_limit=limit)
        with serve.Server(ctx, max_active=4, spp_per_step=8) as srv:
            h = srv.add_scene(*data)
            ids = [srv.submit(h, cam, 128, 128, 8, 4) for _ in range(3)]
            for i in ids:
                assert srv.wait(i, 60000).state == serve.DONE
            images += [srv.image(i).copy() for i in ids]
    assert all(np.array_equal(i, images[0]) for i in images) and images[0].any()


@pytest.mark.parametrize("n", [32, 1000])
def test_no_memory_for_the_cast_tree_leaves_the_references(rt, ctx, tune, n):
    # The cast tree's build takes half a megabyte at least; the scene and its
    # other scratch stay below the limit.
    import torch
    tris, mats = soup(rt, n)
    rays = torch.from_numpy(rt.gen_random_rays(3, 20000, -5, 5)).cuda()
    trees = []
    for limit in (0, 400000):
        tune(test__alloc_limit=limit)
        hits = torch.zeros((len(rays), 4), device="cuda")
        torch.cuda.synchronize()
        sc = ctx.upload_scene(tris, mats)
        sc.trace(rays, len(rays), hits)
        ctx.synchronize()
        trees.append((hits, sc.bvh(), sc.info().device_bytes))
        sc.release()
    assert torch.equal(trees[0][0].view(torch.int32), trees[1][0].view(torch.int32))
    assert np.array_equal(trees[0][1].view(np.uint32), trees[1][1].view(np.uint32)) and trees[0][2] == trees[1][2]
    tune(test__alloc_limit=0, bvh__builder=2)
    ctx.upload_scene(tris, mats).release()
    tune(test__alloc_limit=400000)
    with pytest.raises(rt.RtError):  # the scene's only tree
        ctx.upload_scene(tris, mats)


def test_kept_scratch_is_given_back_when_asked(rt):
    import torch
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    with rt.Context(0) as own:
        assert own.get_tuning("mem.scratch_keep") == 1 << 30
        mats = rt.gen_cornell(1, 0)[1]
        own.upload_scene(rt.gen_icosphere(1, 8), mats).release()
        torch.cuda.synchronize()
        kept = free0 - torch.cuda.mem_get_info()[0]
        own.set_tuning("mem.scratch_keep", 0)
        held = free0 - torch.cuda.mem_get_info()[0]
        assert held < 128 << 20 and held < kept
        own.upload_scene(rt.gen_icosphere(1, 8), mats).release()
        torch.cuda.synchronize()
        assert free0 - torch.cuda.mem_get_info()[0] < 128 << 20
        with pytest.raises(rt.RtError):
            own.set_tuning("mem.scratch_keep", -1)
