"""The GPU build at the sizes where its kernels change over: one CTA per
subtree up to 2,048 triangles, per node up to 16,384, the whole grid above
(ranges of 8,192 and tiles of 4,096), and inputs that use up introsort's
depth limit, so that its heap sort runs in shared and in global memory."""
import numpy as np
import pytest

from test_oracle_pins import _tie_heavy_scene

pytestmark = pytest.mark.gpu

NODE_COLS = [0, 1, 2, 4, 5, 6, 7, 8, 9]


def point_triangles(keys):
    """Degenerate triangles at (k, k, k): every axis sorts by the same keys."""
    t = np.zeros((len(keys), 12), np.float32)
    for c in (0, 1, 2, 4, 5, 6, 8, 9, 10):
        t[:, c] = keys
    return t


def median_killer(n):
    """Keys whose median-of-three partitions split off two elements at a time
    (McIlroy, "A Killer Adversary for Quicksort", 1999), so that introsort
    reaches its depth limit on almost the whole range."""
    order = list(range(n))  # element ids in place
    val = [n] * n  # n: not decided yet
    solid = 0
    last = -1

    def less(a, b):
        nonlocal solid, last
        if val[a] == n and val[b] == n:
            val[a if a == last else b] = solid
            solid += 1
        last = a if val[a] == n else b if val[b] == n else last
        return val[a] < val[b]

    f, l, d = 0, n, 2 * (n.bit_length() - 1)
    while l - f > 16 and d > 0:
        d -= 1
        a, b, c = f + 1, f + (l - f) // 2, l - 1
        if less(order[a], order[b]):
            m = b if less(order[b], order[c]) else c if less(order[a], order[c]) else a
        else:
            m = a if less(order[a], order[c]) else c if less(order[b], order[c]) else b
        order[f], order[m] = order[m], order[f]
        p, lo, hi = order[f], f + 1, l
        while True:
            while less(order[lo], p):
                lo += 1
            hi -= 1
            while less(p, order[hi]):
                hi -= 1
            if not lo < hi:
                break
            order[lo], order[hi] = order[hi], order[lo]
            lo += 1
        f, l = (lo, l) if l - lo > lo - f else (f, lo)
    keys = np.zeros(n, np.float32)
    for i in range(n):
        if val[i] == n:
            val[i] = solid
            solid += 1
        keys[i] = val[i]
    return keys


def check(rt, orc, ctx, tris, seed=1):
    want, depth = orc.build_bvh(tris, seed)
    sc = ctx.upload_scene(tris, rt.gen_cornell(1, 0)[1], bvh_seed=seed)
    try:
        assert np.array_equal(sc.bvh().view(np.uint32)[:, NODE_COLS], want.view(np.uint32)[:, NODE_COLS])
        assert sc.info().depth == depth
    finally:
        sc.release()


@pytest.mark.parametrize("n", [3, 16, 17, 31, 2047, 2048, 2049, 4096, 4098, 8193, 16384, 16385, 32769, 65537, 131075])
def test_changeover_sizes_match_oracle(rt, orc, ctx, n):
    check(rt, orc, ctx, _tie_heavy_scene(n, n), seed=n)


@pytest.mark.parametrize("n", [1500, 12000, 40000])
def test_depth_limit_matches_oracle(rt, orc, ctx, n):
    check(rt, orc, ctx, point_triangles(median_killer(n)))


@pytest.mark.parametrize("n", [2500, 40000])
@pytest.mark.parametrize("order", ["up", "down", "equal"])
def test_ordered_and_equal_keys_match_oracle(rt, orc, ctx, order, n):
    keys = np.arange(n, dtype=np.float32)
    check(rt, orc, ctx, point_triangles(keys if order == "up" else keys[::-1] if order == "down" else 0 * keys))
