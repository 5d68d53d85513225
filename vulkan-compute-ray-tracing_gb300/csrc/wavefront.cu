// Wavefront render: the bounce loop of ray-trace-compute.comp:314-338 split
// into kernels over queues of live paths. A path is one sample of one pixel;
// the samples of a call run together, as many at a time as a wave (kWavePaths) holds.
//
//   camera      closest triangle of every pixel's camera ray, once per call
//               (the ray carries no jitter), 8 x 4 pixel tiles as packets
//   first       per path: record, spheres, scatter of the camera hit with the
//               path's own RNG stream; surviving paths go to the queue
//   per bounce  [Morton reorder of the queue's rays, render.sort] -> closest
//               triangle per ray (the 8-wide caster) -> shade (as above, into
//               the other queue)
//   accumulate  the running mean of comp:375-377, sample by sample
//
// Every floating-point step is the megakernel's (shade.cuh); only the order
// in which paths are processed changes, so images are identical to the
// megakernel's. What the split buys: finished paths leave the queue instead
// of idling lanes, the casting kernel runs without the shading code's
// registers, and each bounce's rays reach the 8-wide caster, whose warps
// refill from the queue (in the order shading queued them, or in Morton
// order when render.sort is set). Queue lengths stay on the device;
// kernels are sized for the queue's capacity and read the live count, so a
// render is a fixed launch sequence (no host synchronisation, capturable in
// a CUDA graph).
#include <cuda_runtime.h>

#include <algorithm>

#include "rt_internal.h"
#include "shade.cuh"

namespace rtgb {
namespace {

constexpr int kWfBlock = 128, kShadeBlock = 256;

// Device words of a wave. Queue lengths and the caster's work counters are
// used in turn; shading clears the ones its next bounce needs.
enum : uint32_t { kCountQueue = 0, kCountWork = 4, kCountWords = 64 };

struct WfBufs {
  rt_ray *rays[2];
  uint32_t *slots[2];
  int2 *hits;
  int2 *cam_hits;  // of the camera rays, by tile position
  float4 *color;
  uint32_t *rng;
  uint32_t *counts;
  void *sort;
};

size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

uint32_t wave_samples(const rt_render_params &p, const Tiles &t, uint32_t wave_paths) {
  return std::max(1u, std::min(p.spp, wave_paths / std::max(t.positions, 1u)));
}

WfBufs carve(void *scratch, uint32_t cap, uint32_t positions) {
  char *p = static_cast<char *>(scratch);
  WfBufs b;
  for (int i = 0; i < 2; i++) {
    b.rays[i] = reinterpret_cast<rt_ray *>(p);
    p += a256(sizeof(rt_ray) * (size_t)cap);
    b.slots[i] = reinterpret_cast<uint32_t *>(p);
    p += a256(4ull * cap);
  }
  b.hits = reinterpret_cast<int2 *>(p);
  p += a256(8ull * cap);
  b.cam_hits = reinterpret_cast<int2 *>(p);
  p += a256(8ull * positions);
  b.color = reinterpret_cast<float4 *>(p);
  p += a256(16ull * cap);
  b.rng = reinterpret_cast<uint32_t *>(p);
  p += a256(4ull * cap);
  b.counts = reinterpret_cast<uint32_t *>(p);
  p += a256(4ull * kCountWords);
  b.sort = p;
  return b;
}

// Sample index of this pass: s, or *d_s + s when the index lives on the
// device (batched jobs advanced by a captured graph).
__device__ __forceinline__ uint32_t sample_of(uint32_t s, const uint32_t *d_s) { return d_s ? *d_s + s : s; }

// Camera rays are packets where triangles are large beside the pixels, and
// rays of their own where a packet's rays soon part: from this many triangles
// a pixel up. us a frame of one sample, packets / own rays: 100K triangles in a
// Cornell box at 2.5 triangles a pixel 1350 / 1360, 1.5 1459 / 1492, 0.1
// 6720 / 7313; a grid mesh of 512K at 12.8 728 / 461, 3.5 1020 / 706, 1.1 1148
// / 957; a finer one of 84M at 200 x 200 14101 / 2005, 1024 x 1000 22057 /
// 13424.
constexpr uint32_t kOwnRayTris = 3;

// The camera rays, a warp per tile: a packet where the tile's rays suit one
// (warp_is_coherent), else each lane's own traversal.
template <int STACK>
__global__ void __launch_bounds__(kWfBlock, 12) k_wf_camera(DevScene sc, rt_camera cam, Tiles tiles,
                                                            int2 *__restrict__ hits, uint32_t *err) {
  const uint32_t pos = blockIdx.x * kWfBlock + threadIdx.x;
  if (pos >= tiles.positions) return;  // whole warps
  uint32_t x, y;
  const bool active = tile_pixel(tiles, pos, x, y);
  const f3 o = ld3(cam.origin);
  const f3 d = active ? normalize3(camera_dir(cam, x, y, tiles.W, tiles.H)) : mk3(1.0f, 0.0f, 0.0f);
  const TraceRay r = make_ray(o, d, kTmin);
  float closest = kTmax, u = 0.0f, v = 0.0f;
  int k;
  const int oct = warp_octant(active, r);
  if (warp_is_coherent(active, r)) {
#define RTGB_CALL(O) k = traverse_packet<STACK, O>(sc, r, active, closest, u, v, err)
    RTGB_OCT_DISPATCH(oct, RTGB_CALL)
#undef RTGB_CALL
  } else {
#define RTGB_CALL(O) k = traverse_spec<STACK, O>(sc, r, active, closest, u, v, err)
    RTGB_OCT_DISPATCH(oct, RTGB_CALL)
#undef RTGB_CALL
  }
  if (active) hits[pos] = make_int2(k, __float_as_int(closest));
}

// The camera rays as a queue for the 8-wide caster; tile positions outside the
// image get a ray of no length.
__global__ void __launch_bounds__(kWfBlock) k_wf_rays(rt_camera cam, Tiles tiles, float4 *__restrict__ rays) {
  const uint32_t pos = blockIdx.x * kWfBlock + threadIdx.x;
  if (pos >= tiles.positions) return;
  uint32_t x, y;
  const bool active = tile_pixel(tiles, pos, x, y);
  const f3 o = ld3(cam.origin);
  const f3 d = active ? normalize3(camera_dir(cam, x, y, tiles.W, tiles.H)) : mk3(1.0f, 0.0f, 0.0f);
  rays[2ull * pos] = make_float4(o.x, o.y, o.z, kTmin);
  rays[2ull * pos + 1] = make_float4(d.x, d.y, d.z, active ? kTmax : -1.0f);
}

// Bounce rays where the 8-wide caster is not used: a warp takes 32 queued
// rays at a time, a packet if they suit one, else each lane its own ray with
// postponed leaves.
template <int STACK>
__global__ void __launch_bounds__(kWfBlock, 12) k_wf_extend(DevScene sc, const float4 *__restrict__ rays,
                                                            uint32_t cap, const uint32_t *count,
                                                            const uint32_t *__restrict__ perm,
                                                            int2 *__restrict__ hits, uint32_t *counter,
                                                            uint32_t *err) {
  const uint32_t n = min(cap, *count);
  const uint32_t lane = threadIdx.x & 31;
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(counter, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n) return;
    uint32_t i = base + lane;
    const bool active = i < n;
    f3 o = mk3(0.0f, 0.0f, 0.0f), d = mk3(1.0f, 0.0f, 0.0f);
    float tmin = 0.0f, closest = 0.0f;
    if (active) {
      if (perm) i = __ldg(perm + i);
      float4 r0 = __ldg(rays + 2ull * i), r1 = __ldg(rays + 2ull * i + 1);
      o = mk3(r0.x, r0.y, r0.z);
      d = mk3(r1.x, r1.y, r1.z);
      tmin = r0.w;
      closest = r1.w;
    }
    TraceRay r = make_ray(o, d, tmin);
    float u = 0.0f, v = 0.0f;
    int k;
    const int oct = warp_octant(active, r);
    if (warp_is_coherent(active, r)) {
#define RTGB_CALL(O) k = traverse_packet<STACK, O>(sc, r, active, closest, u, v, err)
      RTGB_OCT_DISPATCH(oct, RTGB_CALL)
#undef RTGB_CALL
    } else {
#define RTGB_CALL(O) k = traverse_spec<STACK, O>(sc, r, active, closest, u, v, err)
      RTGB_OCT_DISPATCH(oct, RTGB_CALL)
#undef RTGB_CALL
    }
    if (active) hits[i] = make_int2(k, __float_as_int(closest));
  }
}

// Appends the block's surviving paths to the queue, with one atomic a block
// (a warp's own atomic each, on one address, took a third of the shading time).
__device__ __forceinline__ void push_paths(bool push, const HitRec &rec, f3 nd, uint32_t slot, rt_ray *rays_out,
                                           uint32_t *slots_out, uint32_t *count_out) {
  __shared__ uint32_t s_count[kShadeBlock / 32], s_base;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t mask = __ballot_sync(0xffffffffu, push);
  if (lane == 0) s_count[warp] = __popc(mask);
  __syncthreads();
  if (warp == 0) {
    const uint32_t c = lane < kShadeBlock / 32 ? s_count[lane] : 0u;
    const uint32_t total = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0 && total) s_base = atomicAdd(count_out, total);
  }
  __syncthreads();
  if (push) {
    uint32_t pos = s_base + __popc(mask & ((1u << lane) - 1u));
    for (uint32_t w = 0; w < warp; w++) pos += s_count[w];
    rays_out[pos] = rt_ray{{rec.p.x, rec.p.y, rec.p.z}, kTmin, {nd.x, nd.y, nd.z}, kTmax};
    slots_out[pos] = slot;
  }
  __syncthreads();  // the shared words are free again
}

// Shades the first segment of a wave's paths: sample s0 + k of the call at
// tile position q is path (slot) k * positions + q.
__global__ void __launch_bounds__(kShadeBlock) k_wf_first(DevScene sc, uint32_t flags, rt_camera cam, Tiles tiles,
                                                          uint32_t paths, uint32_t s0, const uint32_t *d_s,
                                                          const int2 *__restrict__ hits, float4 *color, uint32_t *rng,
                                                          rt_ray *rays_out, uint32_t *slots_out, uint32_t *count_out,
                                                          int last, unsigned long long *segments) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && segments)
    atomicAdd(segments, (unsigned long long)tiles.W * tiles.H);
  const PathState ps = path_state(sc, flags);
  for (uint32_t base = blockIdx.x * kShadeBlock; base < paths; base += gridDim.x * kShadeBlock) {
    const uint32_t slot = base + threadIdx.x;
    const uint32_t k = slot / tiles.positions, q = slot - k * tiles.positions;
    uint32_t x, y;
    bool push = false;
    HitRec rec;
    f3 nd;
    if (slot < paths && tile_pixel(tiles, q, x, y)) {
      const f3 o = ld3(cam.origin), d = normalize3(camera_dir(cam, x, y, tiles.W, tiles.H));
      const int2 h = hits[q];
      f3 c = mk3(1.0f, 1.0f, 1.0f);
      if (!resolve_hit(sc, ps, o, d, h.x, __int_as_float(h.y), rec)) {
        c = mul3(0.0f, c);
      } else {
        Rng g{(600u * x + y) * (sample_of(s0 + k, d_s) + 1u)};
        f3 albedo;
        const bool emits = scatter(sc, ps, d, rec, g, albedo, nd);
        c = mulv3(c, albedo);
        rng[slot] = g.s;
        push = !emits && !last;
      }
      color[slot] = make_float4(c.x, c.y, c.z, 0.0f);
    }
    push_paths(push, rec, nd, slot, rays_out, slots_out, count_out);
  }
}

__global__ void __launch_bounds__(kShadeBlock) k_wf_shade(DevScene sc, uint32_t flags,
                                                          const rt_ray *__restrict__ rays_in,
                                                          const uint32_t *__restrict__ slots_in, uint32_t cap,
                                                          const uint32_t *count_in, const int2 *__restrict__ hits,
                                                          float4 *color, uint32_t *rng, rt_ray *rays_out,
                                                          uint32_t *slots_out, uint32_t *count_out,
                                                          uint32_t *clear_count, uint32_t *clear_work, int last,
                                                          unsigned long long *segments) {
  const uint32_t n = min(cap, *count_in);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (segments) atomicAdd(segments, (unsigned long long)n);
    *clear_count = 0u;
    *clear_work = 0u;
  }
  const PathState ps = path_state(sc, flags);
  for (uint32_t base = blockIdx.x * kShadeBlock; base < n; base += gridDim.x * kShadeBlock) {
    const uint32_t q = base + threadIdx.x;
    bool push = false;
    HitRec rec;
    f3 nd;
    uint32_t s = 0;
    if (q < n) {
      s = slots_in[q];
      const rt_ray ray = rays_in[q];
      f3 o = ld3(ray.o), d = ld3(ray.d);
      int2 h = hits[q];
      float4 c4 = color[s];
      f3 c = mk3(c4.x, c4.y, c4.z);
      if (!resolve_hit(sc, ps, o, d, h.x, __int_as_float(h.y), rec)) {
        c = mul3(0.0f, c);
      } else {
        Rng g{rng[s]};
        f3 albedo;
        bool emits = scatter(sc, ps, d, rec, g, albedo, nd);
        c = mulv3(c, albedo);
        rng[s] = g.s;
        push = !emits && !last;
      }
      color[s] = make_float4(c.x, c.y, c.z, 0.0f);
    }
    push_paths(push, rec, nd, s, rays_out, slots_out, count_out);
  }
}

// The wave's samples into the running mean, in order. `white`: no bounce was
// asked for, every path's colour is 1.
__global__ void k_wf_accumulate(Tiles tiles, uint32_t s0, uint32_t samples, const uint32_t *d_s, uint32_t flags,
                                bool white, const float4 *__restrict__ color, float4 *accum) {
  const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t x, y;
  if (pos >= tiles.positions || !tile_pixel(tiles, pos, x, y)) return;
  float4 *out = accum + (size_t)y * tiles.W + x;
  float4 acc = *out;
  for (uint32_t k = 0; k < samples; k++) {
    const float4 c = white ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : color[(size_t)k * tiles.positions + pos];
    running_mean(acc, mk3(c.x, c.y, c.z), sample_of(s0 + k, d_s), flags);
  }
  *out = acc;
}

int g_sms = 0;

}  // namespace

size_t wavefront_scratch_bytes(const rt_render_params &p, bool sort, uint32_t wave_paths) {
  const Tiles t = tiles_of(p);
  const size_t cap = (size_t)t.positions * wave_samples(p, t, wave_paths);
  return 2 * (a256(sizeof(rt_ray) * cap) + a256(4 * cap)) + a256(8 * cap) + a256(8ull * t.positions) + a256(16 * cap) +
         a256(4 * cap) + a256(4ull * kCountWords) + (sort ? a256(raysort_scratch_bytes((uint32_t)cap)) : 0);
}

cudaError_t launch_render_wavefront(const DevScene &sc, const rt_camera &cam, const rt_render_params &p, float *accum,
                                    unsigned long long *segments, uint32_t *err, void *scratch,
                                    uint32_t wave_paths, bool sort, bool wide, cudaStream_t st,
                                    const uint32_t *d_sample_index, bool alone) {
  const Tiles tiles = tiles_of(p);
  if (p.width == 0 || p.height == 0 || p.spp == 0) return cudaSuccess;
  const bool use_wide = wide && wide_ok(sc);
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const uint32_t samples = wave_samples(p, tiles, wave_paths), cap = tiles.positions * samples;
  WfBufs b = carve(scratch, cap, tiles.positions);
  uint32_t *queue = b.counts + kCountQueue, *work = b.counts + kCountWork;
  float4 *image = reinterpret_cast<float4 *>(accum);
  const uint32_t tile_grid = (tiles.positions + kWfBlock - 1) / kWfBlock;
  const uint32_t shade_grid = std::min((cap + kShadeBlock - 1) / kShadeBlock, (uint32_t)g_sms * 8u);
  uint32_t extend_grid = 0;
  cudaError_t e = cudaSuccess;
  if (p.max_bounces > 0 && use_wide && sc.ntris / kOwnRayTris >= tiles.positions) {
    if ((e = cudaMemsetAsync(b.counts, 0, 4 * kCountWords, st)) != cudaSuccess) return e;
    k_wf_rays<<<tile_grid, kWfBlock, 0, st>>>(cam, tiles, reinterpret_cast<float4 *>(b.rays[0]));
    const bool pool = alone && tiles.positions <= pool_max_rays(sc);
    if ((e = pool ? launch_pool_leaf(sc, b.rays[0], tiles.positions, nullptr, nullptr, b.cam_hits, work, err, st)
                  : launch_wide_leaf(sc, b.rays[0], tiles.positions, nullptr, nullptr, b.cam_hits, work, err, st)) !=
        cudaSuccess)
      return e;
  } else if (p.max_bounces > 0) {
    if (sc.depth <= 32)
      k_wf_camera<32><<<tile_grid, kWfBlock, 0, st>>>(sc, cam, tiles, b.cam_hits, err);
    else
      k_wf_camera<64><<<tile_grid, kWfBlock, 0, st>>>(sc, cam, tiles, b.cam_hits, err);
  }
  if (p.max_bounces > 1 && !use_wide) {
    int bps = 0;
    if (sc.depth <= 32)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_wf_extend<32>, kWfBlock, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_wf_extend<64>, kWfBlock, 0);
    extend_grid = std::min((uint32_t)(g_sms * std::max(bps, 1)), (cap + kWfBlock - 1) / kWfBlock);
  }
  for (uint32_t k = 0; k < p.spp; k += samples) {
    const uint32_t s0 = d_sample_index ? k : p.sample_index + k, now = std::min(samples, p.spp - k);
    if (p.max_bounces > 0) {
      if ((e = cudaMemsetAsync(b.counts, 0, 4 * kCountWords, st)) != cudaSuccess) return e;
      // The camera segments count once a call.
      k_wf_first<<<shade_grid, kShadeBlock, 0, st>>>(sc, p.flags, cam, tiles, tiles.positions * now, s0,
                                                     d_sample_index, b.cam_hits, b.color, b.rng, b.rays[1],
                                                     b.slots[1], queue + 1, p.max_bounces == 1,
                                                     k == 0 ? segments : nullptr);
    }
    for (uint32_t bounce = 1; bounce < p.max_bounces; bounce++) {
      const int in = bounce & 1, out = in ^ 1;
      const uint32_t *count = queue + bounce % 3;
      uint32_t *perm = nullptr;
      if (sort && (e = launch_raysort(b.rays[in], cap, count, b.sort, &perm, st)) != cudaSuccess) return e;
      if (use_wide) {
        // A short queue of a render that has the GPU to itself is cast from
        // shared pools: one of the two takes the queue, by its length on the
        // device. Beside other renders the pools' extra visits cost more than
        // their shorter chains (a batch of 16 scenes 19.6 ms so, 18.4 without).
        if (alone && (e = launch_pool_leaf(sc, b.rays[in], cap, count, perm, b.hits, work + (bounce & 1), err, st)) !=
                         cudaSuccess)
          return e;
        if ((!alone || cap > pool_max_rays(sc)) &&
            (e = launch_wide_leaf(sc, b.rays[in], cap, count, perm, b.hits, work + (bounce & 1), err, st,
                                  alone ? pool_max_rays(sc) + 1 : 0)) != cudaSuccess)
          return e;
      } else if (sc.depth <= 32) {
        k_wf_extend<32><<<extend_grid, kWfBlock, 0, st>>>(sc, reinterpret_cast<const float4 *>(b.rays[in]), cap,
                                                          count, perm, b.hits, work + (bounce & 1), err);
      } else {
        k_wf_extend<64><<<extend_grid, kWfBlock, 0, st>>>(sc, reinterpret_cast<const float4 *>(b.rays[in]), cap,
                                                          count, perm, b.hits, work + (bounce & 1), err);
      }
      k_wf_shade<<<shade_grid, kShadeBlock, 0, st>>>(
          sc, p.flags, b.rays[in], b.slots[in], cap, count, b.hits, b.color, b.rng, b.rays[out], b.slots[out],
          queue + (bounce + 1) % 3, queue + (bounce + 2) % 3, work + ((bounce + 1) & 1), bounce + 1 == p.max_bounces,
          segments);
    }
    k_wf_accumulate<<<tile_grid, kWfBlock, 0, st>>>(tiles, s0, now, d_sample_index, p.flags, p.max_bounces == 0,
                                                    b.color, image);
  }
  return cudaGetLastError();
}

}  // namespace rtgb
