"""The 8-wide caster's last rays, whose stacks become one pool of nodes: the
same hits, bit for bit, as the casters that do without (one node step per
iteration, a 64-entry stack, the binary layout), on counts around a warp and a
grid of warps, a mesh, and needles that all overlap, whose rays hold more
entries than the pool takes at first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("trace.packet_min_rays", "trace.wide", "trace.wide_visits", "trace.stack", "trace.sort")


def needles(n):
    rng = np.random.default_rng(11)
    t = np.zeros((n, 12), np.float32)
    a = rng.normal(size=(n, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    t[:, 0:3], t[:, 4:7] = a, -a + 0.05 * rng.normal(size=(n, 3))
    t[:, 8:11] = a + 0.002 * rng.normal(size=(n, 3))
    return t


@pytest.fixture(scope="module")
def scenes(rt, ctx):
    mats = rt.gen_cornell(1, 0)[1]
    out = {"mesh": ctx.upload_scene(rt.gen_icosphere(8, 6), mats), "needles": ctx.upload_scene(needles(20011), mats)}
    yield out
    for sc in out.values():
        sc.release()


@pytest.mark.parametrize("name", ["mesh", "needles"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 500, 4097, 70001, 300007])
def test_shared_tail_keeps_hits(rt, ctx, scenes, name, n):
    import torch
    rays = torch.from_numpy(rt.gen_random_rays(21, n)).cuda()
    old = {k: ctx.get_tuning(k) for k in KEYS}

    def cast(**knobs):
        hits = torch.full((n, 4), 7.0, device="cuda")
        torch.cuda.synchronize()
        for k, v in {"packet_min_rays": 0, "sort": 0, **knobs}.items():
            ctx.set_tuning("trace." + k, v)
        try:
            scenes[name].trace(rays, n, hits)
            ctx.synchronize()
        finally:
            for k, v in old.items():
                ctx.set_tuning(k, v)
        return hits.cpu().numpy().view(np.uint32)

    want = cast(wide=0)
    for visits in (1, 2, 3):
        for stack in (0, 32, 64):
            assert np.array_equal(cast(wide_visits=visits, stack=stack), want), (visits, stack)
