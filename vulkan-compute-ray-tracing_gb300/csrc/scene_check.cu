// Checks and light list of an uploaded scene's triangles, on the GPU.
//
// rtUploadScene rejects non-finite vertices and materials out of range, needs
// the largest coordinate (the choice of the tree rays are cast on) and, where
// the caller gives no lights, the triangles of LightSource materials
// (RtScene.h:88-96). One pass over the triangles finds all of it.
#include <cuda_runtime.h>

#include "rt_internal.h"

namespace rtgb {
namespace {

// The triangles as 16-byte words, three a triangle: (v0, pad) (v1, pad)
// (v2, material).
__global__ void k_check_scene(const float4 *__restrict__ tris, uint32_t n, const rt_material *__restrict__ mats,
                              uint32_t nm, SceneCheck *out, uint32_t *__restrict__ lights) {
  const uint32_t lane = threadIdx.x & 31;
  float most = 0.0f;
  uint32_t bad = 0xffffffffu;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    bool light = false;
    if (i < n) {
      const float4 a = __ldg(tris + 3ull * i), b = __ldg(tris + 3ull * i + 1), c = __ldg(tris + 3ull * i + 2);
      const float v[9] = {a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z};
      bool ok = true;
      for (int k = 0; k < 9; k++) {
        ok = ok && isfinite(v[k]);
        most = fmaxf(most, fabsf(v[k]));
      }
      const uint32_t m = __float_as_uint(c.w);
      if (!ok || m >= nm)
        bad = min(bad, i);
      else
        light = mats[m].type == RT_MATERIAL_LIGHT;
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, light);
    if (mask) {
      uint32_t at = 0;
      if (lane == (uint32_t)__ffs(mask) - 1) at = atomicAdd(&out->lights, (uint32_t)__popc(mask));
      at = __shfl_sync(0xffffffffu, at, __ffs(mask) - 1);
      if (light) lights[at + __popc(mask & ((1u << lane) - 1u))] = i;
    }
  }
  const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
  bad = __reduce_min_sync(0xffffffffu, bad);
  if (lane == 0) {
    atomicMax(&out->max_coord, top);
    if (bad != 0xffffffffu) atomicMax(&out->bad, ~bad);
  }
}

}  // namespace

// `out` is zero before the launch; `lights` holds n words and receives the
// light triangles in any order.
cudaError_t launch_check_scene(const rt_triangle *tris, uint32_t n, const rt_material *mats, uint32_t nm,
                               SceneCheck *out, uint32_t *lights, cudaStream_t st) {
  const uint32_t blocks = (n + 255) / 256;
  k_check_scene<<<blocks < 1216 ? blocks : 1216, 256, 0, st>>>(reinterpret_cast<const float4 *>(tris), n, mats, nm,
                                                              out, lights);
  return cudaGetLastError();
}

}  // namespace rtgb
