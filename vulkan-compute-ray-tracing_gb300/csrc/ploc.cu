// Bottom-up agglomerative clustering (PLOC: Meister and Bittner, "Parallel
// Locally-Ordered Clustering for Bounding Volume Hierarchy Construction",
// IEEE TVCG 2018), built on the GPU and emitted in the Bvh.h node layout,
// one triangle per leaf. It is the tree that rays are cast on by default
// ("bvh.cast_tree"), beside the reference's own tree, and the scene's only
// tree with "bvh.builder" = 2.
//
// Triangles start as clusters in Morton order (lbvh.cu's key). Each round,
// every cluster finds, among the `radius` clusters on either side, the one
// whose merged box has the smallest surface area; mutually nearest pairs
// merge into a new inner node; the survivors are compacted in order. Rounds
// repeat until one cluster (the root) is left. The trees approach
// surface-area-heuristic quality, far tighter than the reference's
// random-axis median splits.
//
// All rounds run in one cooperative launch (k_ploc), two grid barriers a
// round; the last clusters are merged by one CTA. Bound by the merged areas
// (32 a cluster and round) in the first rounds, then by latency. Measured:
// 1.4 ms for 1.31M triangles, 0.23 ms for 12K (with a host round trip and
// nine launches a round: 6.7 and 1.3 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>

#include "grid_sync.cuh"
#include "rt_internal.h"

namespace rtgb {

namespace {

// A cluster: box, node id and subtree height, as two 16-byte words.
struct __align__(16) Cluster {
  float lo[3];
  int32_t id;
  float hi[3];
  uint32_t height;
};
// A box in shared memory: two arrays of 16-byte words (no bank conflicts
// between neighbouring clusters).
struct Boxes {
  float4 *lo, *hi;
};

__device__ __forceinline__ Cluster load_cluster(const Cluster *c) {
  const float4 a = __ldcg(reinterpret_cast<const float4 *>(c)), b = __ldcg(reinterpret_cast<const float4 *>(c) + 1);
  return Cluster{{a.x, a.y, a.z}, __float_as_int(a.w), {b.x, b.y, b.z}, __float_as_uint(b.w)};
}
__device__ __forceinline__ void store_cluster(Cluster *c, const Cluster &v) {
  reinterpret_cast<float4 *>(c)[0] = make_float4(v.lo[0], v.lo[1], v.lo[2], __int_as_float(v.id));
  reinterpret_cast<float4 *>(c)[1] = make_float4(v.hi[0], v.hi[1], v.hi[2], __uint_as_float(v.height));
}

__device__ __forceinline__ float joined_area(float4 alo, float4 ahi, float4 blo, float4 bhi) {
  const float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
  const float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
  const float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
  return dx * dy + dy * dz + dz * dx;
}

// Tie key of the unordered pair (i, j), the same seen from either side:
// nearer positions first, then pairs starting at an even position (so that a
// run of equal boxes pairs up as (0, 1), (2, 3), ... and halves each round
// instead of merging one pair per round into a chain), then the lower start.
__device__ __forceinline__ unsigned long long pair_key(uint32_t i, uint32_t j) {
  const uint32_t lo = min(i, j), gap = max(i, j) - lo;
  return ((unsigned long long)gap << 33) | ((unsigned long long)(lo & 1u) << 32) | lo;
}

constexpr int kPlocThreads = 512;
constexpr uint32_t kPlocWarps = kPlocThreads / 32;
constexpr uint32_t kMaxRadius = 256;
// Clusters a CTA handles at a time: with the `radius` beyond them on either
// side, whose nearest it also needs, one a thread where the radius allows.
__host__ __device__ __forceinline__ uint32_t ploc_tile(uint32_t radius) {
  return radius <= kPlocThreads / 4 ? kPlocThreads - 2 * radius : kPlocThreads / 2;
}

// Device words of a build: barrier counter, error bits, clusters left, rounds.
enum : uint32_t { kPlocBarrier = 0, kPlocErr = 1, kPlocLeft = 2, kPlocHeight = 3, kPlocWords = 8 };
enum : uint32_t { kPlocNoProgress = 0x100u };

// What becomes of a cluster: merged with the partner code, kept, or merged
// into a lower partner.
constexpr uint32_t kKeep = 0xffffffffu, kGone = 0xfffffffeu;

// Clusters [t0, t1) of m, at most ploc_tile(radius): their codes, by the boxes
// within 2 * radius of them in shared memory. The nearest neighbour of each
// is the one of least merged area within the radius, equal areas ordered by
// pair_key. Area and key are symmetric in the pair, so the pair smallest in
// (area, key) among all is chosen by both its members: every round merges at
// least one pair. Threads beyond the clusters return kGone.
__device__ uint32_t cluster_code(const Cluster *in, uint32_t m, uint32_t radius, uint32_t t0, uint32_t t1, Boxes s_box,
                                 uint32_t *s_near) {
  const uint32_t b0 = t0 > 2 * radius ? t0 - 2 * radius : 0u, b1 = min(m, t1 + 2 * radius);
  const uint32_t n0 = t0 > radius ? t0 - radius : 0u, n1 = min(m, t1 + radius);
  __syncthreads();
  for (uint32_t i = b0 + threadIdx.x; i < b1; i += kPlocThreads) {
    s_box.lo[i - b0] = __ldcg(reinterpret_cast<const float4 *>(in + i));
    s_box.hi[i - b0] = __ldcg(reinterpret_cast<const float4 *>(in + i) + 1);
  }
  __syncthreads();
  for (uint32_t i = n0 + threadIdx.x; i < n1; i += kPlocThreads) {
    const float4 ilo = s_box.lo[i - b0], ihi = s_box.hi[i - b0];
    float best = __int_as_float(0x7f800000);
    uint32_t arg = i;
    const uint32_t lo = i > radius ? i - radius : 0u, hi = min(m - 1, i + radius);
#pragma unroll 4
    for (uint32_t j = lo; j <= hi; j++) {
      const float a = joined_area(ilo, ihi, s_box.lo[j - b0], s_box.hi[j - b0]);
      if (j != i && (arg == i || a < best || (a == best && pair_key(i, j) < pair_key(i, arg)))) {
        best = a;
        arg = j;
      }
    }
    s_near[i - n0] = arg;
  }
  __syncthreads();
  const uint32_t i = t0 + threadIdx.x;
  if (i >= t1) return kGone;
  const uint32_t j = s_near[i - n0];
  const bool mutual = j != i && s_near[j - n0] == i;
  return !mutual ? kKeep : (i < j ? j : kGone);
}

// Exclusive count of survivors (low half) and merges (high half) before this
// thread, and their totals over the CTA.
__device__ __forceinline__ uint32_t block_count(uint32_t code, uint32_t *s_part, uint32_t &total) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const uint32_t keep = __ballot_sync(0xffffffffu, code != kGone);
  const uint32_t merge = __ballot_sync(0xffffffffu, code < kGone);
  __syncthreads();
  if (lane == 0) s_part[warp] = __popc(keep) | (__popc(merge) << 16);
  __syncthreads();
  const uint32_t v = lane < kPlocWarps ? s_part[lane] : 0u;
  total = __reduce_add_sync(0xffffffffu, v);
  return __reduce_add_sync(0xffffffffu, lane < warp ? v : 0u) + (__popc(keep & lt) | (__popc(merge & lt) << 16));
}

// Writes cluster i's survivor to `out`; a merge's inner node gets number nid.
__device__ __forceinline__ void write_survivor(const Cluster *in, uint32_t i, uint32_t code, Cluster *out, int32_t nid,
                                               rt_bvh_node *nodes) {
  Cluster c = load_cluster(in + i);
  if (code != kKeep) {
    const Cluster d = load_cluster(in + code);
    rt_bvh_node nd;
    for (int k = 0; k < 3; k++) {
      nd.min[k] = c.lo[k] = fminf(c.lo[k], d.lo[k]);
      nd.max[k] = c.hi[k] = fmaxf(c.hi[k], d.hi[k]);
    }
    nd._pad0 = 0.0f;
    nd.left = c.id;
    nd.right = d.id;
    nd.object = -1;
    nd._pad1[0] = nd._pad1[1] = 0;
    nodes[nid] = nd;
    c.id = nid;
    c.height = 1 + max(c.height, d.height);
  }
  store_cluster(out, c);
}

// The whole clustering. Each CTA keeps to one contiguous run of the round's
// clusters: it counts its survivors and merges, then (after a barrier) knows
// the counts of the CTAs before it and writes its survivors in order. Inner
// nodes are numbered down from n - 2, so the last merge is node 0.
__global__ void __launch_bounds__(kPlocThreads) k_ploc(const rt_triangle *__restrict__ tris,
                                                       const uint32_t *__restrict__ idx, uint32_t n, uint32_t radius,
                                                       uint32_t max_rounds, Cluster *buf0, Cluster *buf1,
                                                       uint32_t *codes, uint2 *counts, uint32_t *ctr,
                                                       rt_bvh_node *nodes) {
  extern __shared__ __align__(16) unsigned char s_ploc[];
  const uint32_t tile = ploc_tile(radius);
  Boxes s_box;
  s_box.lo = reinterpret_cast<float4 *>(s_ploc);
  s_box.hi = s_box.lo + tile + 4 * radius;
  uint32_t *s_near = reinterpret_cast<uint32_t *>(s_box.hi + tile + 4 * radius);
  __shared__ uint32_t s_part[kPlocWarps], s_sum[4][kPlocWarps];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t *err = ctr + kPlocErr;
  uint32_t target = 0;
  // Leaves: cluster k = triangle idx[k] in Morton order, node n - 1 + k.
  for (uint32_t k = blockIdx.x * kPlocThreads + tid; k < n; k += gridDim.x * kPlocThreads) {
    const uint32_t o = idx[k];
    const rt_triangle t = tris[o];
    Cluster c;
    rt_bvh_node nd;
    for (int a = 0; a < 3; a++) {
      float lo = (t.v1[a] < t.v0[a]) ? t.v1[a] : t.v0[a];
      lo = (t.v2[a] < lo) ? t.v2[a] : lo;
      float hi = (t.v0[a] < t.v1[a]) ? t.v1[a] : t.v0[a];
      hi = (hi < t.v2[a]) ? t.v2[a] : hi;
      c.lo[a] = nd.min[a] = __fsub_rn(lo, 0.0001f);
      c.hi[a] = nd.max[a] = __fadd_rn(hi, 0.0001f);
    }
    nd._pad0 = 0.0f;
    nd.left = -1;
    nd.right = -1;
    nd.object = (int32_t)o;
    nd._pad1[0] = nd._pad1[1] = 0;
    c.id = (int32_t)(n - 1 + k);
    c.height = 1;
    nodes[n - 1 + k] = nd;
    store_cluster(buf0 + k, c);
  }
  if (!grid_barrier(ctr + kPlocBarrier, err, target)) return;
  uint32_t m = n, round = 0;
  int32_t top = (int32_t)n - 2;
  Cluster *in = buf0, *out = buf1;
  for (; m > tile; round++) {
    if (round >= max_rounds) break;
    const uint32_t run = (m + gridDim.x - 1) / gridDim.x;
    const uint32_t beg = min(m, blockIdx.x * run), end = min(m, beg + run);
    uint32_t keeps = 0, merges = 0;
    for (uint32_t t0 = beg; t0 < end; t0 += tile) {
      const uint32_t t1 = min(end, t0 + tile);
      const uint32_t code = cluster_code(in, m, radius, t0, t1, s_box, s_near);
      if (t0 + tid < t1) codes[t0 + tid] = code;
      uint32_t total;
      block_count(code, s_part, total);
      keeps += total & 0xffffu;
      merges += total >> 16;
    }
    if (tid == 0) counts[blockIdx.x] = make_uint2(keeps, merges);
    if (!grid_barrier(ctr + kPlocBarrier, err, target)) return;
    // Survivors and merges before this CTA, and of the whole round.
    uint32_t v[4] = {0u, 0u, 0u, 0u};
    for (uint32_t b = tid; b < gridDim.x; b += kPlocThreads) {
      const uint2 c = __ldcg(counts + b);
      v[0] += c.x;
      v[1] += c.y;
      if (b < blockIdx.x) {
        v[2] += c.x;
        v[3] += c.y;
      }
    }
    for (int k = 0; k < 4; k++) {
      const uint32_t w = __reduce_add_sync(0xffffffffu, v[k]);
      if (lane == 0) s_sum[k][warp] = w;
    }
    __syncthreads();
    for (int k = 0; k < 4; k++) v[k] = __reduce_add_sync(0xffffffffu, lane < kPlocWarps ? s_sum[k][lane] : 0u);
    uint32_t keep_at = v[2], merge_at = v[3];
    for (uint32_t t0 = beg; t0 < end; t0 += tile) {
      const uint32_t t1 = min(end, t0 + tile);
      const uint32_t code = t0 + tid < t1 ? codes[t0 + tid] : kGone;  // this thread's own write
      uint32_t total;
      const uint32_t before = block_count(code, s_part, total);
      if (code != kGone)
        write_survivor(in, t0 + tid, code, out + keep_at + (before & 0xffffu),
                       top - (int32_t)(merge_at + (before >> 16)), nodes);
      keep_at += total & 0xffffu;
      merge_at += total >> 16;
    }
    top -= (int32_t)v[1];
    if (v[1] == 0 || v[0] + v[1] != m) {
      if (blockIdx.x == 0 && tid == 0) atomicOr(err, kPlocNoProgress);
      return;
    }
    m = v[0];
    Cluster *t = in;
    in = out;
    out = t;
    if (!grid_barrier(ctr + kPlocBarrier, err, target)) return;
  }
  if (blockIdx.x != 0) return;
  // One CTA merges the last tile: a block barrier costs a tenth of a grid barrier.
  for (; m > 1 && round < max_rounds; round++) {
    uint32_t keep_at = 0, merge_at = 0;
    for (uint32_t t0 = 0; t0 < m; t0 += tile) {
      const uint32_t t1 = min(m, t0 + tile);
      const uint32_t code = cluster_code(in, m, radius, t0, t1, s_box, s_near);
      uint32_t total;
      const uint32_t before = block_count(code, s_part, total);
      if (code != kGone)
        write_survivor(in, t0 + tid, code, out + keep_at + (before & 0xffffu),
                       top - (int32_t)(merge_at + (before >> 16)), nodes);
      keep_at += total & 0xffffu;
      merge_at += total >> 16;
    }
    __syncthreads();
    if (merge_at == 0 || keep_at + merge_at != m) {
      if (tid == 0) atomicOr(err, kPlocNoProgress);
      return;
    }
    top -= (int32_t)merge_at;
    m = keep_at;
    Cluster *t = in;
    in = out;
    out = t;
  }
  if (tid == 0) {
    ctr[kPlocLeft] = m;
    ctr[kPlocHeight] = m == 1 ? load_cluster(in).height : 0u;
  }
}

}  // namespace

rt_status gpu_build_ploc(const rt_triangle *d_tris, uint32_t n, uint32_t radius, uint32_t max_rounds,
                         rt_bvh_node *d_nodes, ScratchPool &pool, cudaStream_t st, float *ms_out,
                         uint32_t *depth_out, char *errbuf, size_t errlen) {
  if (n == 0 || radius < 1 || radius > kMaxRadius) return RT_ERR_INVALID_ARGUMENT;
  int dev = 0, sms = 0, per_sm = 0;
  const size_t tile = ploc_tile(radius);
  const size_t smem = 2 * sizeof(float4) * (tile + 4 * radius) + 4 * (tile + 2 * radius);
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ploc, kPlocThreads, smem);
  // Enough CTAs that a run is one tile, and no more: a barrier's cost grows with them.
  const uint32_t grid = std::max(1u, std::min((uint32_t)(sms * std::max(1, std::min(per_sm, 3))),
                                              (uint32_t)((n + tile - 1) / tile)));
  // Scratch, in 32-bit words: the Morton sort | clusters 2 x 8n | codes n |
  // counts 2 x grid | control words.
  const size_t sort_words = (lbvh_sorted_keys_words(n) + 63) & ~size_t(63);
  const size_t words = sort_words + 16ull * n + ((n + 63ull) & ~63ull) + 2ull * grid + 64;
  uint32_t *w = nullptr;
  if (e == cudaSuccess) e = scratch_alloc((void **)&w, 4 * words, pool, st);
  if (e != cudaSuccess) {
    std::snprintf(errbuf, errlen, "ploc scratch: %s", cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? RT_ERR_OUT_OF_MEMORY : RT_ERR_CUDA;
  }
  Cluster *buf0 = reinterpret_cast<Cluster *>(w + sort_words), *buf1 = buf0 + n;
  uint32_t *code = reinterpret_cast<uint32_t *>(buf1 + n);
  uint32_t *ctr = code + ((n + 63ull) & ~63ull);
  uint2 *counts = reinterpret_cast<uint2 *>(ctr + 64);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, st);
  uint32_t *codes = nullptr, *idx = nullptr, *sort_err = nullptr;
  e = lbvh_sorted_keys(d_tris, n, w, &codes, &idx, &sort_err, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ctr, 0, 4 * kPlocWords, st);
  if (e == cudaSuccess) {
    void *args[] = {&d_tris, &idx, &n, &radius, &max_rounds, &buf0, &buf1, &code, &counts, &ctr, &d_nodes};
    e = cudaLaunchCooperativeKernel((const void *)k_ploc, dim3(grid), dim3(kPlocThreads), args, smem, st);
  }
  uint32_t h[kPlocWords] = {0}, sort_bits = 0;
  cudaEventRecord(e1, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, ctr, 4 * kPlocWords, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&sort_bits, sort_err, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  float ms = 0.0f;
  if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
  cudaFreeAsync(w, st);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (e != cudaSuccess) {
    std::snprintf(errbuf, errlen, "ploc build: %s", cudaGetErrorString(e));
    return RT_ERR_CUDA;
  }
  if (h[kPlocErr] || sort_bits || h[kPlocLeft] != 1) {
    std::snprintf(errbuf, errlen, "ploc build: %u clusters left (bits 0x%x)", h[kPlocLeft], h[kPlocErr] | sort_bits);
    return RT_ERR_INTERNAL;
  }
  if (ms_out) *ms_out = ms;
  if (depth_out) *depth_out = h[kPlocHeight];
  return RT_SUCCESS;
}

}  // namespace rtgb
