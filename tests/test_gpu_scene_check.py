"""Upload checks and light lists made on the GPU (scenes of 32,768 triangles
and more) against the host's: the same refusals with the first bad triangle's
number, and the same lights in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def soup(rt, n):
    tris, mats, _ = rt.gen_cornell(n, n)
    return np.ascontiguousarray(tris[12:]), mats


@pytest.mark.parametrize("n", [32767, 32768, 40003])
@pytest.mark.parametrize("word,value", [(0, np.nan), (5, np.inf), (10, -np.inf)])
def test_bad_vertices_are_refused(rt, ctx, n, word, value):
    tris, mats = soup(rt, n)
    for first, second in ((0, n - 1), (n - 1, n - 1), (n // 2, n // 2 + 1)):
        bad = tris.copy()
        bad[second, word] = value
        bad[first, word] = value
        with pytest.raises(rt.RtError) as e:
            ctx.upload_scene(bad, mats)
        assert e.value.status == 5 and f"triangle {first}: non-finite vertex" in str(e.value)


@pytest.mark.parametrize("n", [32767, 32768])
def test_materials_out_of_range_are_refused(rt, ctx, n):
    tris, mats = soup(rt, n)
    for material in (8, 0xffffffff):
        bad = tris.copy()
        bad.view(np.uint32)[777, 11] = material
        with pytest.raises(rt.RtError) as e:
            ctx.upload_scene(bad, mats)
        assert e.value.status == 5 and f"triangle 777: material {material} out of range" in str(e.value)
    sc = ctx.upload_scene(tris, mats)  # and the next upload succeeds
    sc.release()


@pytest.mark.parametrize("n,share", [(32768, 0.0), (32768, 0.3), (50001, 1e-4), (70000, 1.0)])
def test_lights_equal_the_hosts(rt, ctx, n, share):
    tris, mats = soup(rt, n)
    light = int(np.flatnonzero(mats.view(np.uint32)[:, 0] == rt.MATERIAL_LIGHT)[0])
    pick = np.random.RandomState(n).rand(n) < share
    tris.view(np.uint32)[pick, 11] = light
    want = rt.lights_from_materials(tris, mats)
    sc = ctx.upload_scene(tris, mats)
    try:
        got = sc.lights()
        assert len(got) == pick.sum() and np.array_equal(got.view(np.uint32), want.view(np.uint32))
    finally:
        sc.release()
