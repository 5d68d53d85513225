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
                         uint32_t flags) {
  return use_wavefront(opts(mode, pixels), params(w, h, spp, bounces, flags));
}
extern "C" int batched(int mode, uint64_t pixels, uint32_t w, uint32_t h, uint32_t spp, uint32_t flags) {
  return use_wavefront_batched(opts(mode, pixels), params(w, h, spp, 8, flags));
}
extern "C" int fallback(int mode, uint64_t pixels, uint32_t w, uint32_t h) {
  return one_launch_fallback(opts(mode, pixels), params(w, h, 1, 8, 0));
}
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
    lib.wavefront.argtypes = [ctypes.c_int, ctypes.c_uint64, u, u, u, u, u]
    lib.batched.argtypes = [ctypes.c_int, ctypes.c_uint64, u, u, u, u]
    lib.fallback.argtypes = [ctypes.c_int, ctypes.c_uint64, u, u]
    return lib


@pytest.mark.parametrize("spp", [1, 2, 64])
def test_a_threshold_of_the_callers_rules_every_call(routes, spp):
    for pixels in (1, 1 << 10, 1 << 18, 1 << 20):
        side = int(pixels ** 0.5)
        assert routes.wavefront(2, pixels, side, side, spp, 8, 0) == (side * side >= pixels)
        assert not routes.wavefront(2, pixels, side, side - 1, spp, 8, 0)
    for side in (16, 512, 4096):
        assert not routes.wavefront(2, 1 << 31, side, side, spp, 8, 0)  # never


def test_modes_and_flags(routes, rt):
    for side in (8, 600, 2048):
        for spp in (1, 4):
            assert routes.wavefront(1, 0, side, side, spp, 8, 0)
            assert not routes.wavefront(0, 0, side, side, spp, 8, 0)
            assert not routes.wavefront(3, 0, side, side, spp, 8, 0)
            for mode in (0, 1, 2, 3):
                assert not routes.wavefront(mode, 0, side, side, spp, 8, rt.COMPAT_STACK16)
                assert not routes.batched(mode, 0, side, side, spp, rt.COMPAT_STACK16)
            assert [routes.batched(m, 0, side, side, spp, 0) for m in range(4)] == [0, 1, 1, 0]
    assert not routes.batched(2, 1 << 20, 600, 600, 4, 0) and routes.batched(2, 1 << 20, 1024, 1024, 1, 0)


def test_what_falls_back_to_one_launch(routes):
    assert routes.fallback(2, 0, 511, 513) and not routes.fallback(2, 0, 512, 512)
    assert routes.fallback(2, 1 << 31, 4096, 4096) and routes.fallback(2, 1 << 10, 256, 256)
    assert not routes.fallback(1, 0, 64, 64) and not routes.fallback(0, 0, 64, 64)
