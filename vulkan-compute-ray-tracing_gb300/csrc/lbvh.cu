// Alternative tree: a linear BVH over triangle centroids, built on the GPU
// (Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees,
// and k-d Trees", HPG 2012), emitted in the same Bvh.h node layout so the
// re-layout and every traversal kernel run on it unchanged.
//
// The reference's tree splits every node at the median along a random axis
// (Bvh.h:160-175); sibling boxes overlap heavily and a ray visits hundreds of
// nodes. Closest-hit results do not depend on the tree (only the order in
// which equal-t candidates are met does), so this one can be the scene's only
// tree ("bvh.builder" = 1). Its Morton sort also starts the PLOC build
// (ploc.cu), whose tree rays are cast on by default.
//
// Steps: centroid bounds -> 30-bit Morton code per triangle -> stable radix
// sort (k_morton_sort) -> one thread per inner node finds its key range and
// split from the longest common prefixes of neighbouring (code, index) keys
// -> leaves walk to the root with an atomic visit count per inner node; the
// second child to arrive writes the union.
// Leaf boxes are padded by 1e-4 exactly as Bvh.h pads them (Bvh.h:94-98).
#include <cuda_runtime.h>

#include <cstdio>

#include "grid_sync.cuh"
#include "rt_internal.h"

namespace rtgb {
namespace {

__device__ __forceinline__ uint32_t f2o(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ float3 centroid(const rt_triangle &t) {
  return make_float3((t.v0[0] + t.v1[0] + t.v2[0]) * (1.0f / 3.0f), (t.v0[1] + t.v1[1] + t.v2[1]) * (1.0f / 3.0f),
                     (t.v0[2] + t.v1[2] + t.v2[2]) * (1.0f / 3.0f));
}

constexpr int kSortThreads = 512;
constexpr uint32_t kSortWarps = kSortThreads / 32;
constexpr uint32_t kSortPer = 8;                             // keys a lane holds at most
constexpr uint32_t kSortMaxGrid = 512;
constexpr uint32_t kRadix = 256;

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v &= 1023u;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}


// Morton codes of the centroids and their stable radix sort, in one
// cooperative launch: centroid bounds; codes; four 8-bit passes, each a
// digit histogram per CTA (over its contiguous run of keys), a scan of each
// digit's row over the CTAs, and the scatter, a grid barrier apart. Within a
// tile a warp ranks equal digits with match_any, in order, and the warps'
// counts are prefixed per digit. Latency-bound (12 barriers). A run is short
// (512 keys) rather than the grid small where there are few keys. Measured:
// 0.17 ms for 1.31M triangles, 0.04 ms for 12K (one-bit passes of five
// launches each: 1.0 and 0.4 ms).
//   sync: barrier counter, error bits, then the ordered bounds (6 words)
//   rows: kRadix x gridDim.x counts, then kRadix totals
__global__ void __launch_bounds__(kSortThreads) k_morton_sort(const rt_triangle *__restrict__ tris, uint32_t n,
                                                              uint32_t *sync, uint32_t *codes0, uint32_t *codes1,
                                                              uint32_t *idx0, uint32_t *idx1, uint32_t *rows) {
  __shared__ uint32_t s_warp[kSortWarps][kRadix], s_base[kRadix], s_part[kSortWarps];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
  uint32_t *err = sync + 1, *ext = sync + 2, *totals = rows + kRadix * gridDim.x;
  uint32_t target = 0;
  // Each CTA keeps to one run of keys, `per` a lane at a time.
  const uint32_t run = (n + gridDim.x - 1) / gridDim.x;
  const uint32_t per = min(kSortPer, (run + kSortThreads - 1) / kSortThreads), tile = per * kSortThreads;
  const uint32_t beg = (uint32_t)min((uint64_t)blockIdx.x * run, (uint64_t)n);
  const uint32_t end = min(n, beg + run);
  {
    float lo[3] = {3.4e38f, 3.4e38f, 3.4e38f}, hi[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (uint32_t i = beg + tid; i < end; i += kSortThreads) {
      const float3 c = centroid(tris[i]);
      lo[0] = fminf(lo[0], c.x), lo[1] = fminf(lo[1], c.y), lo[2] = fminf(lo[2], c.z);
      hi[0] = fmaxf(hi[0], c.x), hi[1] = fmaxf(hi[1], c.y), hi[2] = fmaxf(hi[2], c.z);
    }
    for (int k = 0; k < 3; k++) {
      const uint32_t a = __reduce_min_sync(0xffffffffu, f2o(lo[k])), b = __reduce_max_sync(0xffffffffu, f2o(hi[k]));
      if (lane == 0) {
        atomicMin(ext + k, a);
        atomicMax(ext + 3 + k, b);
      }
    }
  }
  if (!grid_barrier(sync, err, target)) return;
  float lo[3], span[3];
  for (int k = 0; k < 3; k++) {
    lo[k] = o2f(__ldcg(ext + k));
    span[k] = o2f(__ldcg(ext + 3 + k)) - lo[k];
  }
  for (uint32_t i = beg + tid; i < end; i += kSortThreads) {
    const float3 c = centroid(tris[i]);
    const float p[3] = {c.x, c.y, c.z};
    uint32_t q[3];
    for (int k = 0; k < 3; k++) {
      float t = span[k] > 0.0f ? (p[k] - lo[k]) / span[k] : 0.0f;
      t = fminf(fmaxf(t, 0.0f), 1.0f);
      q[k] = min(1023u, (uint32_t)(t * 1024.0f));
    }
    codes0[i] = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
    idx0[i] = i;
  }
  for (int pass = 0; pass < 4; pass++) {
    const uint32_t *ci = pass & 1 ? codes1 : codes0, *vi = pass & 1 ? idx1 : idx0;
    uint32_t *co = pass & 1 ? codes0 : codes1, *vo = pass & 1 ? idx0 : idx1;
    const int shift = 8 * pass;
    __syncthreads();  // pass 0: the codes of this CTA's run (its own writes)
    for (uint32_t d = tid; d < kRadix; d += kSortThreads) s_base[d] = 0u;
    __syncthreads();
    for (uint32_t i = beg + tid; i < end; i += kSortThreads) atomicAdd(&s_base[(__ldcg(ci + i) >> shift) & 255u], 1u);
    __syncthreads();
    for (uint32_t d = tid; d < kRadix; d += kSortThreads) rows[d * gridDim.x + blockIdx.x] = s_base[d];
    if (!grid_barrier(sync, err, target)) return;
    // Rows: exclusive prefix over the CTAs and the total, a warp each.
    for (uint32_t d = blockIdx.x * kSortWarps + warp; d < kRadix; d += gridDim.x * kSortWarps) {
      uint32_t before = 0;
      for (uint32_t b0 = 0; b0 < gridDim.x; b0 += 32) {
        const uint32_t v = b0 + lane < gridDim.x ? __ldcg(rows + d * gridDim.x + b0 + lane) : 0u;
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= (uint32_t)o) x += y;
        }
        if (b0 + lane < gridDim.x) rows[d * gridDim.x + b0 + lane] = before + x - v;
        before += __shfl_sync(0xffffffffu, x, 31);
      }
      if (lane == 0) totals[d] = before;
    }
    if (!grid_barrier(sync, err, target)) return;
    // This CTA's first slot per digit: the smaller digits, then its column of the digit's row.
    if (tid < kRadix) {
      const uint32_t v = __ldcg(totals + tid);
      uint32_t x = v;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      if (lane == 31) s_part[warp] = x;
      s_base[tid] = x - v + __ldcg(rows + tid * gridDim.x + blockIdx.x);
    }
    __syncthreads();
    if (tid < kRadix) {
      uint32_t before = 0;
      for (uint32_t w = 0; w < warp; w++) before += s_part[w];
      s_base[tid] += before;
    }
    for (uint32_t t0 = beg; t0 < end; t0 += tile) {
      for (uint32_t d = tid; d < kSortWarps * kRadix; d += kSortThreads) (&s_warp[0][0])[d] = 0u;
      __syncthreads();
      uint32_t c[kSortPer], v[kSortPer], rank[kSortPer];
      const uint32_t w0 = t0 + warp * (32 * per);
#pragma unroll
      for (uint32_t j = 0; j < kSortPer; j++) {
        const uint32_t i = w0 + j * 32 + lane;
        c[j] = j < per && i < end ? __ldcg(ci + i) : 0u;
        v[j] = j < per && i < end ? __ldcg(vi + i) : 0u;
      }
#pragma unroll
      for (uint32_t j = 0; j < kSortPer; j++) {
        if (j >= per) continue;
        const bool in = w0 + j * 32 + lane < end;
        const uint32_t d = in ? (c[j] >> shift) & 255u : kRadix;  // lanes past the end match only one another
        const uint32_t same = __match_any_sync(0xffffffffu, d);
        const uint32_t at = in ? s_warp[warp][d] : 0u;
        __syncwarp();
        if (in && (same & lt) == 0) s_warp[warp][d] = at + __popc(same);
        __syncwarp();
        rank[j] = at + __popc(same & lt);
      }
      __syncthreads();
      if (tid < kRadix) {
        uint32_t at = s_base[tid];
        for (uint32_t w = 0; w < kSortWarps; w++) {
          const uint32_t m = s_warp[w][tid];
          s_warp[w][tid] = at;
          at += m;
        }
        s_base[tid] = at;
      }
      __syncthreads();
#pragma unroll
      for (uint32_t j = 0; j < kSortPer; j++) {
        if (j >= per || w0 + j * 32 + lane >= end) continue;
        const uint32_t at = s_warp[warp][(c[j] >> shift) & 255u] + rank[j];
        co[at] = c[j];
        vo[at] = v[j];
      }
      __syncthreads();
    }
    if (pass < 3 && !grid_barrier(sync, err, target)) return;
  }
}

// Longest common prefix of the keys (code, position) at i and j; -1 outside.
__device__ __forceinline__ int delta(const uint32_t *codes, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint32_t a = codes[i], b = codes[j];
  if (a != b) return __clz(a ^ b);
  return 32 + __clz((uint32_t)i ^ (uint32_t)j);
}

__global__ void k_karras(const uint32_t *__restrict__ codes, int n, int32_t *left, int32_t *right, int32_t *parent) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (delta(codes, n, i, i + 1) - delta(codes, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = delta(codes, n, i, i - d);
  int lmax = 2;
  while (delta(codes, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(codes, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = delta(codes, n, i, j);
  int s = 0;
  for (int t = (l + 1) >> 1;; t = (t + 1) >> 1) {
    if (delta(codes, n, i, i + (s + t) * d) > dnode) s += t;
    if (t == 1) break;
  }
  int g = i + s * d + (d < 0 ? -1 : 0);
  int lo = i < j ? i : j, hi = i < j ? j : i;
  // Inner nodes are 0..n-2, leaf k is node n-1+k.
  int L = (lo == g) ? (n - 1 + g) : g;
  int R = (hi == g + 1) ? (n - 1 + g + 1) : (g + 1);
  left[i] = L;
  right[i] = R;
  parent[L] = i;
  parent[R] = i;
}

// Node read that bypasses L1: the sibling wrote it from another SM.
__device__ __forceinline__ void load_box_cg(const rt_bvh_node *nd, float lo[3], float hi[3]) {
  const float4 *p = reinterpret_cast<const float4 *>(nd);
  float4 a = __ldcg(p), b = __ldcg(p + 1);
  lo[0] = a.x;
  lo[1] = a.y;
  lo[2] = a.z;
  hi[0] = b.x;
  hi[1] = b.y;
  hi[2] = b.z;
}

constexpr int kMaxWalk = 128;  // longer than any path of a 30-bit-code LBVH (<= 64 levels)

__global__ void k_lbvh_boxes(const rt_triangle *__restrict__ tris, const uint32_t *__restrict__ idx, int n,
                             const int32_t *__restrict__ left, const int32_t *__restrict__ right,
                             const int32_t *__restrict__ parent, uint32_t *visits, rt_bvh_node *nodes,
                             uint32_t *depth_max) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int leaf = n - 1 + k;
  const uint32_t o = idx[k];
  const rt_triangle t = tris[o];
  rt_bvh_node nd;
  for (int a = 0; a < 3; a++) {
    float lo = (t.v1[a] < t.v0[a]) ? t.v1[a] : t.v0[a];
    lo = (t.v2[a] < lo) ? t.v2[a] : lo;
    float hi = (t.v0[a] < t.v1[a]) ? t.v1[a] : t.v0[a];
    hi = (hi < t.v2[a]) ? t.v2[a] : hi;
    nd.min[a] = __fsub_rn(lo, 0.0001f);
    nd.max[a] = __fadd_rn(hi, 0.0001f);
  }
  nd._pad0 = 0.0f;
  nd.left = -1;
  nd.right = -1;
  nd.object = (int32_t)o;
  nd._pad1[0] = nd._pad1[1] = 0;
  nodes[leaf] = nd;
  int cur = leaf;
  for (int step = 0; cur != 0; step++) {
    int p = parent[cur];
    if (step >= kMaxWalk || p < 0 || p >= n - 1) {
      atomicMax(depth_max, 0xffffffffu);  // malformed: reported as an error by the host
      return;
    }
    __threadfence();
    if (atomicAdd(visits + p, 1u) == 0) break;  // the sibling finishes the parent
    __threadfence();
    float alo[3], ahi[3], blo[3], bhi[3];
    load_box_cg(nodes + left[p], alo, ahi);
    load_box_cg(nodes + right[p], blo, bhi);
    rt_bvh_node q;
    for (int c = 0; c < 3; c++) {
      q.min[c] = fminf(alo[c], blo[c]);
      q.max[c] = fmaxf(ahi[c], bhi[c]);
    }
    q._pad0 = 0.0f;
    q.left = left[p];
    q.right = right[p];
    q.object = -1;
    q._pad1[0] = q._pad1[1] = 0;
    nodes[p] = q;
    cur = p;
  }
  // Levels on this leaf's path (root = 1).
  uint32_t levels = 1;
  for (int c = leaf, step = 0; c != 0 && step < kMaxWalk; c = parent[c], step++) levels++;
  atomicMax(depth_max, levels);
}

}  // namespace

size_t lbvh_sorted_keys_words(uint32_t n) { return 64 + 4ull * n + kRadix * (kSortMaxGrid + 1); }

// Centroid bounds -> Morton codes -> stable radix sort. `scratch` holds
// lbvh_sorted_keys_words(n) words: barrier, error bits and bounds 64 | codes
// 2n | indices 2n | digit rows. The sorted codes and triangle indices are
// returned as pointers into it.
cudaError_t lbvh_sorted_keys(const rt_triangle *d_tris, uint32_t n, uint32_t *scratch, uint32_t **codes_out,
                             uint32_t **idx_out, uint32_t **err_out, cudaStream_t st) {
  uint32_t *sync = scratch, *codes0 = scratch + 64, *codes1 = codes0 + n, *idx0 = codes1 + n, *idx1 = idx0 + n;
  uint32_t *rows = idx1 + n;
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_morton_sort, kSortThreads, 0);
  if (e == cudaSuccess) e = cudaMemsetAsync(sync, 0, 4 * 64, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(sync + 2, 0xff, 4 * 3, st);  // lower bounds
  if (e != cudaSuccess) return e;
  const uint32_t grid =
      min(min((uint32_t)sms * (uint32_t)max(1, min(per_sm, 2)), kSortMaxGrid), (n + kSortThreads - 1) / kSortThreads);
  void *args[] = {&d_tris, &n, &sync, &codes0, &codes1, &idx0, &idx1, &rows};
  e = cudaLaunchCooperativeKernel((const void *)k_morton_sort, dim3(grid), dim3(kSortThreads), args, 0, st);
  *codes_out = codes0;  // four passes: back in the first pair
  *idx_out = idx0;
  *err_out = sync + 1;
  return e;
}

rt_status gpu_build_lbvh(const rt_triangle *d_tris, uint32_t n, rt_bvh_node *d_nodes, ScratchPool &pool,
                         cudaStream_t st, float *ms_out, uint32_t *depth_out, char *errbuf, size_t errlen) {
  if (n == 0) return RT_ERR_INVALID_ARGUMENT;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  // Scratch, in 32-bit words: the sort's words | left n | right n |
  // parent 2n | visit counts n | depth 8.
  void *mem = nullptr;
  const size_t sort_words = lbvh_sorted_keys_words(n);
  const size_t words = sort_words + n + n + 2ull * n + n + 8;
  cudaError_t e = scratch_alloc(&mem, 4 * words, pool, st);
  if (e != cudaSuccess) {
    std::snprintf(errbuf, errlen, "lbvh scratch: %s", cudaGetErrorString(e));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return RT_ERR_OUT_OF_MEMORY;
  }
  uint32_t *sortbuf = static_cast<uint32_t *>(mem);
  int32_t *left = reinterpret_cast<int32_t *>(sortbuf + sort_words);
  int32_t *right = left + n;
  int32_t *parent = right + n;
  uint32_t *visits = reinterpret_cast<uint32_t *>(parent + 2ull * n);
  uint32_t *dmax = visits + n;
  cudaEventRecord(e0, st);
  const uint32_t B = 256, G = (n + B - 1) / B;
  uint32_t *codes = nullptr, *idx = nullptr, *sort_err = nullptr;
  e = lbvh_sorted_keys(d_tris, n, sortbuf, &codes, &idx, &sort_err, st);
  if (e == cudaSuccess) {
    cudaMemsetAsync(visits, 0, 4ull * n + 32, st);  // visit counts and the depth word
    cudaMemsetAsync(parent, 0xff, 4ull * 2 * n, st);
    if (n > 1) k_karras<<<(n - 1 + B - 1) / B, B, 0, st>>>(codes, (int)n, left, right, parent);
    k_lbvh_boxes<<<G, B, 0, st>>>(d_tris, idx, (int)n, left, right, parent, visits, d_nodes, dmax);
  }
  cudaEventRecord(e1, st);
  uint32_t depth = 0, sort_bits = 0;
  cudaMemcpyAsync(&depth, dmax, 4, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&sort_bits, sortbuf + 1, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  float ms = 0.0f;
  if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
  cudaFreeAsync(mem, st);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (e != cudaSuccess) {
    std::snprintf(errbuf, errlen, "lbvh build: %s", cudaGetErrorString(e));
    return RT_ERR_CUDA;
  }
  if (depth == 0xffffffffu || depth == 0 || sort_bits) {
    std::snprintf(errbuf, errlen, "lbvh build: malformed tree");
    return RT_ERR_INTERNAL;
  }
  if (ms_out) *ms_out = ms;
  if (depth_out) *depth_out = depth;
  return RT_SUCCESS;
}

}  // namespace rtgb
