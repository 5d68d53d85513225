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
