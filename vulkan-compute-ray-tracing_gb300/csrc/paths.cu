// Small one-sample renders in one persistent launch: a warp follows R paths at
// a time, each from the camera ray to its last bounce, and traverses their
// segments from its shared pools (pool.cuh).
//
// A slot whose ray is done waits until a few are (kShadeAt) or the pools are
// empty; those lanes then shade together: record, spheres, scatter, and either
// the bounce ray or the end of the path, whose colour goes into the running
// mean. Free slots claim the next pixels, in 8 x 4 tiles. The hit rule is every
// traversal's and shading is shade.cuh's, so the image is every other form's,
// bit for bit.
//
// An image that does not fill the GPU takes as long as its longest path's
// chain of node and leaf steps; side by side in the pool that chain is several
// times shorter than a thread's own (k_render). us, megakernel / R = 4 / R = 8:
// 48 x 48 in a 12K-triangle Cornell box 647 / 164 / 254, in 1.31M triangles
// 5610 / 518 / 923; 256 x 256 762 / 945 / 733 and 5187 / 2038 / 1923; 512 x 512
// (2272 / 3496 / 2541) is a wavefront's, 1725.
#include <cuda_runtime.h>

#include <algorithm>

#include "rt_internal.h"
#include "pool.cuh"
#include "shade.cuh"

namespace rtgb {
namespace {

constexpr int kShadeAt = 4, kClaimAt = 2;

template <int R>
struct PathsWarp {
  PoolWarp<R> pool;
  float4 path[R];  // colour and RNG state
};

template <int R, int MINB>
__global__ void __launch_bounds__(kPoolBlock, MINB) k_paths(DevScene sc, rt_camera cam, Tiles tiles,
                                                             uint32_t max_bounces, uint32_t sample, uint32_t flags,
                                                             float4 *__restrict__ accum,
                                                             unsigned long long *segments, uint32_t *counter,
                                                             uint32_t *err) {
  extern __shared__ float4 s_paths[];
  uint32_t lane;
  asm("mov.u32 %0, %%laneid;" : "=r"(lane));
  const uint32_t lt_mask = (1u << lane) - 1u;
  PathsWarp<R> &W = reinterpret_cast<PathsWarp<R> *>(s_paths)[threadIdx.x >> 5];
  PoolWarp<R> &S = W.pool;
  volatile PoolWarp<R> &V = S;
  if (lane == 0) S.node_count = S.leaf_tail = 0u;
  __syncwarp();
  const unsigned long long key_miss = pool_miss_key(kTmax);
  const PathState ps = path_state(sc, flags);

  int pos = -1;  // of lanes < R: the tile position of the path in their slot
  uint32_t bounce = 0, segs = 0, head = 0;
  bool exhausted = false;
  for (;;) {
    // Rays with nothing left in the pools.
    const bool room = V.node_count <= kNodeRoom;
    const bool ready = pos >= 0 && V.left[lane % R] == 0u;
    const uint32_t rm = __ballot_sync(0xffffffffu, ready), am = __ballot_sync(0xffffffffu, pos >= 0);
    if (room && rm && (__popc(rm) >= min(kShadeAt, R) || rm == am)) {
      if (ready) {
        const unsigned long long key = V.key[lane];
        const float4 h = S.hit[lane], q0 = S.org[lane], q1 = S.dir[lane], pc = W.path[lane];
        const bool got = (uint32_t)(key >> 32) != (uint32_t)(key_miss >> 32);
        const f3 o = mk3(q0.x, q0.y, q0.z), d = mk3(q1.x, q1.y, q1.z);
        f3 c = mk3(pc.x, pc.y, pc.z), nd = d;
        Rng g{__float_as_uint(pc.w)};
        HitRec rec;
        bool on = false;
        if (!resolve_hit(sc, ps, o, d, got ? __float_as_int(h.w) : -1, got ? h.x : kTmax, rec)) {
          c = mul3(0.0f, c);
        } else {
          f3 albedo;
          const bool emits = scatter(sc, ps, d, rec, g, albedo, nd);
          c = mulv3(c, albedo);
          on = !emits && ++bounce < max_bounces;
        }
        if (on) {
          W.path[lane] = make_float4(c.x, c.y, c.z, __uint_as_float(g.s));
          pool_start(S, sc, lane, rec.p, nd, kTmin, kTmax);
          segs++;
        } else {
          uint32_t x, y;
          tile_pixel(tiles, (uint32_t)pos, x, y);
          float4 acc = accum[(size_t)y * tiles.W + x];
          running_mean(acc, c, sample, flags);
          accum[(size_t)y * tiles.W + x] = acc;
          pos = -1;
        }
      }
    }
    // Slots without a path claim pixels.
    const uint32_t idle = __ballot_sync(0xffffffffu, pos < 0 && lane < R);
    if (room && !exhausted && __popc(idle) >= kClaimAt) {
      const uint32_t cnt = __popc(idle), leader = __ffs(idle) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(counter, cnt);
      base = __shfl_sync(0xffffffffu, base, leader);
      if (base + cnt >= tiles.positions) exhausted = true;
      const uint32_t at = base + __popc(idle & lt_mask);
      uint32_t x, y;
      if (pos < 0 && lane < R && at < tiles.positions && tile_pixel(tiles, at, x, y)) {
        pos = (int)at;
        bounce = 0;
        W.path[lane] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float((600u * x + y) * (sample + 1u)));
        pool_start(S, sc, lane, ld3(cam.origin), normalize3(camera_dir(cam, x, y, tiles.W, tiles.H)), kTmin, kTmax);
        segs++;
      }
    }
    if (exhausted && __all_sync(0xffffffffu, pos < 0)) break;
    __syncwarp();

    pool_step(S, sc, lane, head, err);
  }
  segs = __reduce_add_sync(0xffffffffu, segs);
  if (lane == 0 && segments) atomicAdd(segments, (unsigned long long)segs);
}

int g_sms = 0;

template <int R, int MINB>
cudaError_t go(const DevScene &sc, const rt_camera &cam, const rt_render_params &p, float *accum,
               unsigned long long *segments, uint32_t *counter, uint32_t *err, cudaStream_t st) {
  auto kern = k_paths<R, MINB>;
  const size_t smem = (size_t)(kPoolBlock / 32) * sizeof(PathsWarp<R>);
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPoolBlock, smem);
  if (e == cudaSuccess) e = cudaMemsetAsync(counter, 0, 4, st);
  if (e != cudaSuccess) return e;
  const Tiles t = tiles_of(p);
  const uint32_t grid = std::min((uint32_t)(g_sms * std::max(per_sm, 1)), (t.positions + kPoolBlock / 32 * R - 1) / (kPoolBlock / 32 * R));
  kern<<<grid, kPoolBlock, smem, st>>>(sc, cam, t, p.max_bounces, p.sample_index, p.flags,
                                        reinterpret_cast<float4 *>(accum), segments, counter, err);
  return cudaGetLastError();
}

}  // namespace

bool paths_ok(const DevScene &sc, const rt_render_params &p) {
  return wide_ok(sc) && p.spp == 1 && p.max_bounces > 0 && !(p.flags & RT_COMPAT_STACK16) && paths_fit(sc.ntris, p);
}

cudaError_t launch_render_paths(const DevScene &sc, const rt_camera &cam, const rt_render_params &p, float *accum,
                                unsigned long long *segments, uint32_t *counter, uint32_t *err, cudaStream_t st) {
  if (p.width == 0 || p.height == 0 || p.spp == 0) return cudaSuccess;
  if (!paths_ok(sc, p)) return cudaErrorInvalidValue;
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  // Few paths a warp while the grid has room for all of them, else more.
  const uint32_t positions = tiles_of(p).positions;
  if (positions <= 8192) return go<2, 4>(sc, cam, p, accum, segments, counter, err, st);
  if (positions <= 24576) return go<4, 4>(sc, cam, p, accum, segments, counter, err, st);
  return go<8, 6>(sc, cam, p, accum, segments, counter, err, st);
}

}  // namespace rtgb
