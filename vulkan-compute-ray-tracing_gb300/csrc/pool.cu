// Closest hits of small batches: R rays a warp from its shared pools
// (pool.cuh). Free slots claim the batch's next rays; a finished ray's hit is
// written by its slot's lane, re-evaluated in fp64 when asked for.
#include <cuda_runtime.h>

#include <algorithm>

#include "pool.cuh"
#include "refine.cuh"
#include "rt_internal.h"

namespace rtgb {
namespace {

// LEAF_OUT: hits are int2 (leaf k, fp32 t) for the wavefront's shading, and the
// batch is the first *d_n rays, left to k_trace_wide when more than max_rays;
// otherwise int4 rt_hit records.
template <int R, int MINB, bool LEAF_OUT>
__global__ void __launch_bounds__(kPoolBlock, MINB) k_trace_pool(DevScene sc, const float4 *__restrict__ rays,
                                                                 uint32_t n, const uint32_t *d_n, uint32_t max_rays,
                                                                 const uint32_t *__restrict__ perm,
                                                                 void *__restrict__ hits_out, uint32_t *counter,
                                                                 uint32_t *err, bool refine) {
  extern __shared__ float4 s_pool[];
  if (d_n) n = min(n, *d_n);
  if (n > max_rays) return;
  uint32_t lane;
  asm("mov.u32 %0, %%laneid;" : "=r"(lane));
  PoolWarp<R> &S = reinterpret_cast<PoolWarp<R> *>(s_pool)[threadIdx.x >> 5];
  volatile PoolWarp<R> &V = S;
  if (lane == 0) S.node_count = S.leaf_tail = 0u;
  __syncwarp();
  int ray = -1;  // of lanes < R: the ray in their slot
  uint32_t head = 0;
  bool exhausted = false;
  for (;;) {
    const bool room = V.node_count <= kNodeRoom;
    if (ray >= 0 && V.left[lane % R] == 0u) {
      const unsigned long long key = V.key[lane];
      const float tmax = S.inv[lane].w;
      const bool got = (uint32_t)(key >> 32) != (uint32_t)(pool_miss_key(tmax) >> 32);
      const float4 h = S.hit[lane];
      if (LEAF_OUT) {
        static_cast<int2 *>(hits_out)[ray] =
            got ? make_int2(__float_as_int(h.w), __float_as_int(h.x)) : make_int2(-1, __float_as_int(tmax));
      } else {
        int4 out = make_int4(-1, 0, 0, 0);
        if (got) {
          const int tri = (int)(uint32_t)key;
          const float4 o = S.org[lane], d = S.dir[lane];
          float t = h.x, u = h.y, v = h.z;
          if (refine) refine_fp64(sc.tris, tri, mk3(o.x, o.y, o.z), mk3(d.x, d.y, d.z), t, u, v);
          out = make_int4(tri, __float_as_int(t), __float_as_int(u), __float_as_int(v));
        }
        static_cast<int4 *>(hits_out)[ray] = out;
      }
      ray = -1;
    }
    const uint32_t idle = __ballot_sync(0xffffffffu, ray < 0 && lane < R);
    if (room && !exhausted && idle) {
      const uint32_t cnt = __popc(idle), leader = __ffs(idle) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(counter, cnt);
      base = __shfl_sync(0xffffffffu, base, leader);
      if (base + cnt >= n) exhausted = true;
      const uint32_t at = base + __popc(idle & ((1u << lane) - 1u));
      if (ray < 0 && lane < R && at < n) {
        const uint32_t i = perm ? __ldg(perm + at) : at;
        const float4 r0 = __ldg(rays + 2ull * i), r1 = __ldg(rays + 2ull * i + 1);
        ray = (int)i;
        pool_start(S, sc, lane, mk3(r0.x, r0.y, r0.z), mk3(r1.x, r1.y, r1.z), r0.w, r1.w);
      }
    }
    if (exhausted && __all_sync(0xffffffffu, ray < 0)) return;
    __syncwarp();
    pool_step(S, sc, lane, head, err);
  }
}

int g_sms = 0;

template <int R, int MINB, bool LEAF_OUT>
cudaError_t go(const DevScene &sc, const rt_ray *rays, uint32_t n, const uint32_t *d_n, uint32_t max_rays,
               const uint32_t *perm, void *hits, uint32_t *counter, uint32_t *err, bool refine, cudaStream_t st) {
  auto kern = k_trace_pool<R, MINB, LEAF_OUT>;
  const size_t smem = (size_t)(kPoolBlock / 32) * sizeof(PoolWarp<R>);
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPoolBlock, smem);
  if (e != cudaSuccess) return e;
  const uint32_t block_rays = kPoolBlock / 32 * R, most = std::min(n, max_rays);
  const uint32_t grid = std::min((uint32_t)(g_sms * std::max(per_sm, 1)), (most + block_rays - 1) / block_rays);
  kern<<<grid, kPoolBlock, smem, st>>>(sc, reinterpret_cast<const float4 *>(rays), n, d_n, max_rays, perm, hits,
                                       counter, err, refine);
  return cudaGetLastError();
}

void init_sms() {
  if (g_sms != 0) return;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
}

}  // namespace

cudaError_t launch_trace_pool(const DevScene &sc, const rt_ray *rays, uint32_t n, rt_hit *hits, uint32_t *counter,
                              uint32_t *err, bool refine, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (!wide_ok(sc)) return cudaErrorInvalidValue;
  init_sms();
  const cudaError_t e = cudaMemsetAsync(counter, 0, 4, st);
  if (e != cudaSuccess) return e;
  // Two rays a warp as long as that many warps run at once, then four. us, 8,000
  // / 16,384 random rays, two / four: into 20K triangles 33 / 32 and 47 / 43, into
  // 1.31M 80 / 99 and 104 / 117.
  if (n <= 8192) return go<2, 4, false>(sc, rays, n, nullptr, n, nullptr, hits, counter, err, refine, st);
  return go<4, 4, false>(sc, rays, n, nullptr, n, nullptr, hits, counter, err, refine, st);
}

cudaError_t launch_pool_leaf(const DevScene &sc, const rt_ray *rays, uint32_t cap, const uint32_t *d_n,
                             const uint32_t *perm, int2 *hits, uint32_t *counter, uint32_t *err, cudaStream_t st) {
  if (!wide_ok(sc)) return cudaErrorInvalidValue;
  init_sms();
  return go<4, 4, true>(sc, rays, cap, d_n, pool_max_rays(sc), perm, hits, counter, err, false, st);
}

}  // namespace rtgb
