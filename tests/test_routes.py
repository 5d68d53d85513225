"""The rules that choose a call's kernels by its sizes (csrc/routes.h), on the CPU."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG, ROOT

SRC = r"""
#include "routes.h"
using namespace rtgb;
static rt_render_params params(uint32_t w, uint32_t h, uint32_t spp, uint32_t bounces, uint32_t flags) {
  rt_render_params p{};
  p.width = w, p.height = h, p.spp = spp, p.max_bounces = bounces, p.flags = flags;
  return p;
}
static RenderOpts opts(int mode, uint64_t pixels) {
  RenderOpts o;
  o.mode = mode;
  if (pixels) o.wavefront_pixels = o.batch_wavefront_pixels = pixels;
  return o;
}
extern "C" int wavefront(int mode, uint64_t pixels, uint32_t w, uint32_t h, uint32_t spp, uint32_t bounces,
                         uint32_t flags, uint32_t ntris) {
  return use_wavefront(opts(mode, pixels), ntris, params(w, h, spp, bounces, flags));
}
extern "C" int paths(uint32_t ntris, uint32_t w, uint32_t h, uint32_t bounces) {
  return paths_fit(ntris, params(w, h, 1, bounces, 0));
}
extern "C" int batched(int mode, uint64_t pixels, uint32_t w, uint32_t h, uint32_t spp, uint32_t flags) {
  return use_wavefront_batched(opts(mode, pixels), params(w, h, spp, 8, flags));
}
extern "C" int fallback(int mode, uint64_t pixels, uint32_t w, uint32_t h) {
  return one_launch_fallback(opts(mode, pixels), params(w, h, 1, 8, 0));
}
extern "C" int direct(uint32_t ntris, uint32_t n, uint32_t line) { return direct_rays(ntris, n, line, false); }
extern "C" int chunk(uint32_t ntris, uint32_t n, uint32_t line) { return direct_rays(ntris, n, line, true); }
"""


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    d = tmp_path_factory.mktemp("routes")
    src, so = d / "routes.cpp", d / "routes.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(ROOT, "include"), str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    u = ctypes.c_uint32
    lib.wavefront.argtypes = [ctypes.c_int, ctypes.c_uint64, u, u, u, u, u, u]
    lib.batched.argtypes = [ctypes.c_int, ctypes.c_uint64, u, u, u, u]
    lib.fallback.argtypes = [ctypes.c_int, ctypes.c_uint64, u, u]
    return lib


@pytest.mark.parametrize("spp", [1, 2, 64])
def test_a_threshold_of_the_callers_rules_every_call(routes, spp):
    for pixels in (1, 1 << 10, 1 << 18, 1 << 20):
        side = int(pixels ** 0.5)
        assert routes.wavefront(2, pixels, side, side, spp, 8, 0, 12) == (side * side >= pixels)
        assert not routes.wavefront(2, pixels, side, side - 1, spp, 8, 0, 12)
    for side in (16, 512, 4096):
        assert not routes.wavefront(2, 1 << 31, side, side, spp, 8, 0, 12)  # never


def test_modes_and_flags(routes, rt):
    for side in (8, 600, 2048):
        for spp in (1, 4):
            assert routes.wavefront(1, 0, side, side, spp, 8, 0, 12)
            assert not routes.wavefront(0, 0, side, side, spp, 8, 0, 12)
            assert not routes.wavefront(3, 0, side, side, spp, 8, 0, 12)
            for mode in (0, 1, 2, 3):
                assert not routes.wavefront(mode, 0, side, side, spp, 8, rt.COMPAT_STACK16, 12)
                assert not routes.batched(mode, 0, side, side, spp, rt.COMPAT_STACK16)
            assert [routes.batched(m, 0, side, side, spp, 0) for m in range(4)] == [0, 1, 1, 0]
    assert not routes.batched(2, 1 << 20, 600, 600, 4, 0) and routes.batched(2, 1 << 20, 1024, 1024, 1, 0)


def test_what_falls_back_to_one_launch(routes):
    assert routes.fallback(2, 0, 511, 513) and not routes.fallback(2, 0, 512, 512)
    assert routes.fallback(2, 1 << 31, 4096, 4096) and routes.fallback(2, 1 << 10, 256, 256)
    assert not routes.fallback(1, 0, 64, 64) and not routes.fallback(0, 0, 64, 64)


def test_small_scenes_keep_the_megakernel(routes):
    # Few triangles, bounces or rows: a wavefront's launches and a pool's steps cost more than they save.
    for side in (1, 8, 64, 128, 256, 300, 380, 511):
        for spp in (1, 2, 3):
            assert not routes.wavefront(2, 0, side, side, spp, 8, 0, 12)
            assert not routes.wavefront(2, 0, side, side, spp, 8, 0, 320)
        assert not routes.paths(12, side, side, 8) and not routes.paths(20, side, side, 1)
    assert not routes.wavefront(2, 0, 256, 256, 2, 1, 0, 1012)
    assert not routes.wavefront(2, 0, 4096, 1, 4, 8, 0, 12012) and not routes.wavefront(2, 0, 1, 1, 2, 8, 0, 12012)
    assert not routes.paths(112, 128, 128, 8) and not routes.paths(1012, 256, 256, 4) and not routes.paths(5120, 256, 256, 3)
    assert not routes.paths(12012, 1, 65536, 8) and not routes.paths(12012, 1, 1, 8)
    assert not routes.wavefront(2, 0, 1, 1, 16, 8, 0, 1 << 20) and not routes.wavefront(2, 0, 1, 4096, 4, 4, 0, 320)


def test_larger_scenes_keep_their_waves_and_paths(routes):
    for ntris in (1000, 12012, 100012, 1 << 20):
        for spp in (2, 4, 64):
            for w, h in ((48, 48), (500, 375), (256, 256), (1024, 48), (511, 513)):
                assert routes.wavefront(2, 0, w, h, spp, 2, 0, ntris) and routes.wavefront(2, 0, w, h, spp, 8, 0, ntris)
        assert routes.wavefront(2, 0, 362, 363, 1, 8, 0, ntris) and not routes.wavefront(2, 0, 362, 362, 1, 8, 0, ntris)
        for side in (3, 48, 128, 181, 256):
            assert routes.paths(ntris, side, side, 8)
        assert routes.paths(ntris, 256, 256, 2) == (ntris >= 10000)
        assert routes.paths(ntris, 512, 128, 1) and not routes.paths(ntris, 128, 513, 8)
    for ntris in (1, 12, 320, 1 << 20):  # from 2^18 pixels up, and many samples
        assert routes.wavefront(2, 0, 512, 512, 1, 1, 0, ntris) and routes.wavefront(2, 0, 64, 64, 64, 8, 0, ntris)
    assert not routes.paths(1 << 20, 257, 256, 8)


def test_batches_that_are_cast_as_they_are(routes):
    line = 1 << 20
    for ntris in (1, 1280, 9999, 100000, 327680, 1 << 19):
        assert routes.direct(ntris, line - 1, line) and not routes.direct(ntris, line, line)
    for ntris in (10000, 20480, 81920, 99999):  # packets pay sooner
        assert routes.direct(ntris, 917503, line) and not routes.direct(ntris, 917504, line)
    for ntris in (1310720, 2048012):  # and later where triangles outnumber the rays
        assert routes.direct(ntris, 3 * ntris // 2 - 1, line) and not routes.direct(ntris, 3 * ntris // 2, line)
        assert routes.chunk(ntris, line - 1, line) and not routes.chunk(ntris, line, line)  # not beside other casts
    for ntris in (1, 20480, 1 << 30):
        assert not routes.direct(ntris, 1, 0)  # 0: never
        assert routes.direct(ntris, 0xf0000000, 0xffffffff) == (not 10000 <= ntris < 100000)
