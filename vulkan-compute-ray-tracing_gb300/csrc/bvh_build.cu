// GPU BVH build, node-for-node identical to Bvh::createBvh
// (src/ray-tracing/Bvh.h:141-209).
//
// What the reference does, and what decides each output word:
//   * Topology. A node with n triangles gets n/2 on the left and the rest on
//     the right (Bvh.h:175-197); the DFS stack pops the right child first and
//     the creation counter names children 2k+1 / 2k+2 when the k-th inner
//     node is popped (Bvh.h:178-192). So indices, child links and the order
//     in which nodes draw rand() depend on n alone: pop rank of the right
//     child = parent + 1, of the left child = parent + 2*|right|; inner
//     rank = pop rank - leaves popped before (child_item).
//   * Axis. rand() % 3 once per popped node, leaves included (Bvh.h:160):
//     glibc's sequence (glibc_rand.cpp), drawn by k_axes.
//   * Which triangles a child receives, and in what order, is the sorted
//     order of its parent's triangles under std::sort (Bvh.h:166) with the
//     key min(v0,v1,v2)[axis] - 1e-4 (Bvh.h:94-98,116-122). Ties are common,
//     so the sort is replayed exactly (sort_emul.cuh).
//   * Boxes are unions of padded triangle boxes (Bvh.h:94-114); min/max are
//     order-free on finite values, so they are computed bottom-up at the end.
//
// GPU organisation. All triangles live in one array `idx`; a node owns the
// slice [off, off+n), and sorting a node in place leaves its children's
// slices in their input order. A node's slice, indices and draw follow from
// its path alone (item_below), so no kernel reads a node table. The build runs
// level by level from the root:
//   1. Levels whose nodes exceed kSegCap (k_big_level): one cooperative grid
//      partitions every range of the level at once, a round per introsort
//      step, until all ranges are small; k_sort_queue finishes those, one
//      CTA each.
//   2. Levels of kTreeCap to kSegCap (k_sort_segs): one CTA sorts one node.
//   3. From kTreeCap down (k_subtrees): one CTA sorts every level of one
//      subtree, then writes its leaves and inner boxes bottom-up; k_top joins
//      the boxes above.
// In 1-3 the CTA works on keys and indices in shared memory (block_sort).
// An introsort partition is done in parallel: the swap pairs of an unguarded
// Hoare partition are the i-th "!(x < p)" from the left and the i-th
// "!(p < x)" from the right; the cut is min(P[K], Q[K-1]) for the K pairs
// that have not crossed. Ranges of at most 16 get the stable order the final
// insertion sort gives them, by rank; heap sort where the depth limit runs out.
//
// What bounds it: the chain of partition steps (about 1.5 log2(n) dependent
// rounds per level, each a few hundred cycles of latency), not bandwidth: all
// arrays stay in L2 or shared memory. Measured, 1.31M triangles: 4.2 ms (big
// levels 2.2, their queues 1.0, node sorts 0.4, subtrees 0.6) against 54 ms
// with a CTA per node and warps sorting in global memory; 12,012 triangles:
// 0.3 against 4.6 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "grid_sync.cuh"
#include "rt_internal.h"
#include "sort_emul.cuh"

namespace rtgb {
namespace {

constexpr uint32_t kTreeCap = 2048;    // largest subtree one CTA builds
constexpr uint32_t kRangeCap = 8192;   // largest range of a big level that one CTA finishes
constexpr uint32_t kSegCap = 16384;    // largest node one CTA sorts (12 B an element: 197 KB of shared memory)
constexpr uint32_t kWarpRange = 2048;  // largest range one warp partitions
constexpr uint32_t kInsertion = 16;    // libstdc++'s threshold: smaller ranges are left to the insertion sort
constexpr uint32_t kTile = 4096;       // elements of a range that one CTA of a big level handles at a time
constexpr int kBigThreads = 512;
constexpr int kMaxRounds = 128;        // a depth limit of 2 log2(n) ends every sort long before

struct Range {
  uint32_t f, l, d;
};
// A range of a big level being partitioned: its first tile and, after the
// counting pass, how many elements are !(x < p) and !(p < x).
struct BigRange {
  uint32_t f, l, d, tile0, ge, le;
};

// A node of the tree by its path: slice, node number, pop rank and leaves
// popped before it.
struct Item {
  uint32_t off, n, node, rank, leaves;
};
__host__ __device__ __forceinline__ Item root_item(uint32_t n) { return Item{0u, n, 0u, 0u, 0u}; }
__host__ __device__ __forceinline__ Item child_item(const Item &it, bool right) {
  const uint32_t k = it.rank - it.leaves, nl = it.n / 2, nr = it.n - nl;
  return right ? Item{it.off + nl, nr, 2 * k + 2, it.rank + 1, it.leaves}
               : Item{it.off, nl, 2 * k + 1, it.rank + 2 * nr, it.leaves + nr};
}
// Node i (of 2^level, left to right) of a level below `it`.
__device__ __forceinline__ Item item_below(Item it, uint32_t level, uint32_t i) {
  for (uint32_t b = level; b > 0; b--) it = child_item(it, (i >> (b - 1)) & 1u);
  return it;
}
// The node `level` levels below `it` whose slice holds position e.
__device__ __forceinline__ Item item_holding(Item it, uint32_t level, uint32_t e) {
  for (uint32_t b = 0; b < level; b++) it = child_item(it, e >= it.off + it.n / 2);
  return it;
}
// Largest node of the level (halving rounds up): all 2^level nodes exist
// while this is at least 2.
__host__ __device__ __forceinline__ uint32_t level_max(uint32_t n, uint32_t level) {
  return (uint32_t)(((uint64_t)n + (1ull << level) - 1) >> level);
}

__device__ __forceinline__ float tri_key(const rt_triangle &t, int axis) {
  float a = t.v0[axis], b = t.v1[axis], c = t.v2[axis];
  float m = (b < a) ? b : a;
  m = (c < m) ? c : m;
  return __fsub_rn(m, 0.0001f);
}

// The 2n - 1 draws, kAxisRun a warp. A warp multiplies the powers of its
// run's start (polynomials of 31 coefficients, one a lane), applies the
// product to the first words, and continues the recurrence 30 words a step:
// r[i] = r[i-3] + r[i-31], ten times, is r[i-30] + sum_{j<10} r[i-31-3j].
// 2.6M draws in 0.02 ms; the host's loop took 4.8 ms.
constexpr int kAxisWarps = 8;
constexpr uint32_t kAxisRun = 1u << AxisJump::kRunLog2;
__global__ void __launch_bounds__(32 * kAxisWarps) k_axes(AxisJump jump, uint64_t count, uint8_t *__restrict__ axes) {
  __shared__ uint32_t s_word[kAxisWarps][kAxisRun + 64], s_a[kAxisWarps][32], s_b[kAxisWarps][32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t run = (uint64_t)blockIdx.x * kAxisWarps + warp;
  if (run * kAxisRun >= count) return;
  uint32_t *a = s_a[warp], *b = s_b[warp], *w = s_word[warp];
  uint32_t c = lane == 0 ? 1u : 0u;  // the product so far: 1
  for (int bit = 0; bit < AxisJump::kPowers; bit++) {
    if (!((run >> bit) & 1u)) continue;
    a[lane] = lane < 31 ? c : 0u;
    b[lane] = lane < 31 ? jump.pow2[bit][lane] : 0u;
    __syncwarp();
    // Coefficients lane and 31 + lane of the product.
    uint32_t lo = 0, hi = 0;
    for (uint32_t i = 0; i < 31; i++) {
      if (lane >= i) lo += a[i] * b[lane - i];
      if (31 + lane - i < 31) hi += a[i] * b[31 + lane - i];
    }
    // x^(31+m) = x^(28+m) + x^m: of the high coefficients, H[m] = h[m] + H[m+3].
    if (lane >= 30) hi = 0;
    for (int s = 3; s < 32; s <<= 1) {
      const uint32_t up = __shfl_down_sync(0xffffffffu, hi, s);
      if (lane + s < 32) hi += up;
    }
    const uint32_t low3 = __shfl_sync(0xffffffffu, hi, (lane + 4) & 31);  // H[lane - 28] for lanes 28 to 30
    c = lo + hi + (lane >= 28 ? low3 : 0u);
    if (lane >= 31) c = 0;
    __syncwarp();
  }
  // The run's first 31 words.
  a[lane] = c;
  __syncwarp();
  uint32_t v = 0;
  if (lane < 31)
    for (uint32_t k = 0; k < 31; k++) v += a[k] * jump.first[k + lane];
  if (lane < 31) w[lane] = v;
  __syncwarp();
  // The next 30 one by one (three at a time), then 30 a step.
  for (uint32_t i = 31; i < 61; i += 3) {
    if (lane < 3) w[i + lane] = w[i + lane - 3] + w[i + lane - 31];
    __syncwarp();
  }
  for (uint32_t i = 61; i < kAxisRun + 31; i += 30) {
    if (lane < 30) {
      uint32_t r = w[i + lane - 30];
      for (uint32_t j = 0; j < 10; j++) r += w[i + lane - 31 - 3 * j];
      w[i + lane] = r;
    }
    __syncwarp();
  }
  const uint64_t base = run * kAxisRun;
  for (uint32_t k = lane; k < kAxisRun && base + k < count; k += 32) axes[base + k] = (uint8_t)((w[31 + k] >> 1) % 3u);
}

// Test hook of the build's error word: records `bits` as a sort kernel
// would on an overflow, so a test can check that an error raised at any
// level survives to the end of the build.
__global__ void k_flag_error(uint32_t *err, uint32_t bits) { atomicOr(err, bits); }

// Every vertex coordinate must be finite: the sort replay orders keys with
// IEEE `<`, which a NaN key breaks, and node boxes are min/max unions. Any
// non-finite coordinate sets `bits` in the error word.
__global__ void k_check_finite(const rt_triangle *__restrict__ tris, uint32_t n, uint32_t *err, uint32_t bits) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const rt_triangle t = tris[i];
  bool ok = true;
  for (int k = 0; k < 3; k++) ok = ok && isfinite(t.v0[k]) && isfinite(t.v1[k]) && isfinite(t.v2[k]);
  if (!ok) atomicOr(err, bits);
}

// Which of (a, mid, c) median_to_first moves to the front.
__device__ __forceinline__ uint32_t median_of(float ka, float kb, float kc, uint32_t a, uint32_t b, uint32_t c) {
  if (ka < kb) return kb < kc ? b : (ka < kc ? c : a);
  return ka < kc ? a : (kb < kc ? c : b);
}

// ------------------------------------------------- sorting in shared memory
template <int CAP, int NT>
struct SortSmem {
  float key[CAP];
  uint32_t idx[CAP];
  // Rank lists of the partition under way: of a range [f, l), P[f + j] is
  // its j-th !(x < p) and Q[f + j] its j-th !(p < x), both from the left. Of
  // a finished range of at most kInsertion: P = f, Q = l for each element.
  uint16_t P[CAP], Q[CAP];
  // Ranges above kInsertion of this round and the next: f | l << 16, depth.
  uint32_t list[2][CAP / 16];
  uint8_t depth[2][CAP / 16];
  uint32_t count[2], big_count[2];
  uint32_t big[2][CAP / kWarpRange + 1];  // those above kWarpRange, partitioned by the whole CTA
  uint8_t big_depth[2][CAP / kWarpRange + 1];
  uint32_t warp_ge[32], warp_le[32];
};

// Adds a range to the next round's list, or marks it finished; called by
// the lanes of one warp with the same arguments.
template <int CAP, int NT>
__device__ __forceinline__ void push_range(SortSmem<CAP, NT> &S, int next, uint32_t f, uint32_t l, uint32_t d,
                                           uint32_t lane, uint32_t *err) {
  const uint32_t n = l - f;
  if (n <= kInsertion) {
    if (lane < n) {
      S.P[f + lane] = (uint16_t)f;
      S.Q[f + lane] = (uint16_t)l;
    }
  } else if (lane == 0) {
    if (CAP > (int)kWarpRange && n > kWarpRange) {
      const uint32_t k = atomicAdd(&S.big_count[next], 1u);
      if (k > CAP / kWarpRange) {
        atomicOr(err, KERR_STACK_OVERFLOW);
        return;
      }
      S.big[next][k] = f | (l << 16);
      S.big_depth[next][k] = (uint8_t)d;
    } else {
      const uint32_t k = atomicAdd(&S.count[next], 1u);
      if (k >= CAP / 16) {
        atomicOr(err, KERR_STACK_OVERFLOW);
        return;
      }
      S.list[next][k] = f | (l << 16);
      S.depth[next][k] = (uint8_t)d;
    }
  }
}

// The K swap pairs of a partition: the count of j < m with P[j] < Q[le-1-j]
// (true, then false). Each warp searches by itself, 32 probes a step.
__device__ __forceinline__ uint32_t count_pairs(const uint16_t *P, const uint16_t *Q, uint32_t m, uint32_t le,
                                                uint32_t lane) {
  uint32_t lo = 0, hi = m;
  while (lo < hi) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t j = lo + (lane + 1) * step - 1;
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, j < hi && P[j] < Q[le - 1 - j]));
    lo += c * step;
    hi = min(hi, lo + step - 1);
  }
  return lo;
}

template <int CAP, int NT>
__device__ __forceinline__ void swap_pairs(SortSmem<CAP, NT> &S, uint32_t f, uint32_t le, uint32_t K, uint32_t first,
                                           uint32_t stride) {
  for (uint32_t j = first; j < K; j += stride) {
    const uint32_t a = S.P[f + j], b = S.Q[f + le - 1 - j];
    const float ka = S.key[a], kb = S.key[b];
    const uint32_t va = S.idx[a], vb = S.idx[b];
    S.key[a] = kb;
    S.idx[a] = vb;
    S.key[b] = ka;
    S.idx[b] = va;
  }
}

template <int CAP, int NT>
__device__ __forceinline__ uint32_t cut_of(const SortSmem<CAP, NT> &S, uint32_t f, uint32_t ge, uint32_t le,
                                           uint32_t K) {
  uint32_t cut = K < ge ? S.P[f + K] : 0xffffffffu;
  if (K >= 1) cut = min(cut, (uint32_t)S.Q[f + le - K]);
  return cut;
}

// One warp's partition of [f, l) (more than kInsertion elements).
template <int CAP, int NT>
__device__ __forceinline__ uint32_t warp_partition(SortSmem<CAP, NT> &S, uint32_t f, uint32_t l, uint32_t lane) {
  const uint32_t lt = (1u << lane) - 1u, mid = f + (l - f) / 2;
  const float kf = S.key[f], ka = S.key[f + 1], kb = S.key[mid], kc = S.key[l - 1];
  const uint32_t m = median_of(ka, kb, kc, f + 1, mid, l - 1);
  const float pk = m == mid ? kb : (m == f + 1 ? ka : kc);
  __syncwarp();
  if (lane == 0) {
    const uint32_t vf = S.idx[f];
    S.key[f] = pk;
    S.idx[f] = S.idx[m];
    S.key[m] = kf;
    S.idx[m] = vf;
  }
  __syncwarp();
  uint32_t ge = 0, le = 0;
  for (uint32_t base = f + 1; base < l; base += 32) {
    const uint32_t i = base + lane;
    const float k = i < l ? S.key[i] : 0.0f;
    const bool g = i < l && !(k < pk), e = i < l && !(pk < k);
    const uint32_t bg = __ballot_sync(0xffffffffu, g), be = __ballot_sync(0xffffffffu, e);
    if (g) S.P[f + ge + __popc(bg & lt)] = (uint16_t)i;
    if (e) S.Q[f + le + __popc(be & lt)] = (uint16_t)i;
    ge += __popc(bg);
    le += __popc(be);
  }
  __syncwarp();
  const uint32_t K = count_pairs(S.P + f, S.Q + f, min(ge, le), le, lane);
  const uint32_t cut = cut_of(S, f, ge, le, K);
  swap_pairs(S, f, le, K, lane, 32u);
  __syncwarp();
  return cut;
}

// The whole CTA's partition: warp w takes the w-th run of elements.
template <int CAP, int NT>
__device__ __forceinline__ uint32_t cta_partition(SortSmem<CAP, NT> &S, uint32_t f, uint32_t l) {
  constexpr uint32_t NW = NT / 32;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, mid = f + (l - f) / 2;
  const float kf = S.key[f], ka = S.key[f + 1], kb = S.key[mid], kc = S.key[l - 1];
  const uint32_t m = median_of(ka, kb, kc, f + 1, mid, l - 1);
  const float pk = m == mid ? kb : (m == f + 1 ? ka : kc);
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t vf = S.idx[f];
    S.key[f] = pk;
    S.idx[f] = S.idx[m];
    S.key[m] = kf;
    S.idx[m] = vf;
  }
  __syncthreads();
  const uint32_t chunk = ((l - f - 1 + NW - 1) / NW + 31) & ~31u;
  const uint32_t beg = min(l, f + 1 + warp * chunk), end = min(l, beg + chunk);
  uint32_t ge = 0, le = 0;
  for (uint32_t base = beg; base < end; base += 32) {
    const uint32_t i = base + lane;
    const float k = i < end ? S.key[i] : 0.0f;
    ge += __popc(__ballot_sync(0xffffffffu, i < end && !(k < pk)));
    le += __popc(__ballot_sync(0xffffffffu, i < end && !(pk < k)));
  }
  if (lane == 0) {
    S.warp_ge[warp] = ge;
    S.warp_le[warp] = le;
  }
  __syncthreads();
  const uint32_t wg = lane < NW ? S.warp_ge[lane] : 0u, we = lane < NW ? S.warp_le[lane] : 0u;
  const uint32_t ge_all = __reduce_add_sync(0xffffffffu, wg), le_all = __reduce_add_sync(0xffffffffu, we);
  ge = __reduce_add_sync(0xffffffffu, lane < warp ? wg : 0u);
  le = __reduce_add_sync(0xffffffffu, lane < warp ? we : 0u);
  for (uint32_t base = beg; base < end; base += 32) {
    const uint32_t i = base + lane;
    const float k = i < end ? S.key[i] : 0.0f;
    const bool g = i < end && !(k < pk), e = i < end && !(pk < k);
    const uint32_t bg = __ballot_sync(0xffffffffu, g), be = __ballot_sync(0xffffffffu, e);
    if (g) S.P[f + ge + __popc(bg & lt)] = (uint16_t)i;
    if (e) S.Q[f + le + __popc(be & lt)] = (uint16_t)i;
    ge += __popc(bg);
    le += __popc(be);
  }
  __syncthreads();
  const uint32_t K = count_pairs(S.P + f, S.Q + f, min(ge_all, le_all), le_all, lane);
  const uint32_t cut = cut_of(S, f, ge_all, le_all, K);
  swap_pairs(S, f, le_all, K, threadIdx.x, (uint32_t)NT);
  __syncthreads();
  return cut;
}

// Runs the listed ranges (list[0], big[0]) through introsort's partition
// steps, a round at a time, until only finished ranges of at most kInsertion
// are left; ranges whose depth limit runs out are heap-sorted and each of
// their elements marked finished. Called by the whole CTA after a barrier.
template <int CAP, int NT>
__device__ void block_sort(SortSmem<CAP, NT> &S, uint32_t *err) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int cur = 0;
  for (int round = 0; round < kMaxRounds; round++) {
    __syncthreads();
    const uint32_t cnt = min(S.count[cur], (uint32_t)(CAP / 16));
    const uint32_t nbig = CAP > (int)kWarpRange ? min(S.big_count[cur], (uint32_t)(CAP / kWarpRange + 1)) : 0u;
    if (cnt + nbig == 0) break;
    if (threadIdx.x == 0) S.count[cur ^ 1] = S.big_count[cur ^ 1] = 0;
    __syncthreads();
    for (int r = 0; r < (int)nbig; r++) {
      const uint32_t e = S.big[cur][r], f = e & 0xffffu, l = e >> 16, d = S.big_depth[cur][r];
      if (d == 0) {
        if (threadIdx.x == 0) sortemu::heap_sort(S.key + f, S.idx + f, (long)(l - f));
        for (uint32_t i = f + threadIdx.x; i < l; i += NT) S.P[i] = (uint16_t)i, S.Q[i] = (uint16_t)(i + 1);
        __syncthreads();
        continue;
      }
      const uint32_t cut = cta_partition(S, f, l);
      if (cut <= f || cut >= l) {  // cannot happen for finite keys: the median guards both scans
        if (threadIdx.x == 0) atomicOr(err, KERR_BAD_INDEX);
        for (uint32_t i = f + threadIdx.x; i < l; i += NT) S.P[i] = (uint16_t)i, S.Q[i] = (uint16_t)(i + 1);
        __syncthreads();
        continue;
      }
      if (warp == 0) {
        push_range(S, cur ^ 1, f, cut, d - 1, lane, err);
        push_range(S, cur ^ 1, cut, l, d - 1, lane, err);
      }
      // The next cta_partition's first barrier orders its writes after these.
    }
    for (uint32_t r = warp; r < cnt; r += NT / 32) {
      const uint32_t e = S.list[cur][r], f = e & 0xffffu, l = e >> 16, d = S.depth[cur][r];
      uint32_t cut = f;
      if (d > 0) {
        cut = warp_partition(S, f, l, lane);
        if (cut <= f || cut >= l) {
          if (lane == 0) atomicOr(err, KERR_BAD_INDEX);
          cut = f;
        }
      } else {
        if (lane == 0) sortemu::heap_sort(S.key + f, S.idx + f, (long)(l - f));
        __syncwarp();
      }
      if (cut == f) {
        for (uint32_t i = f + lane; i < l; i += 32) S.P[i] = (uint16_t)i, S.Q[i] = (uint16_t)(i + 1);
      } else {
        push_range(S, cur ^ 1, f, cut, d - 1, lane, err);
        push_range(S, cur ^ 1, cut, l, d - 1, lane, err);
      }
    }
    cur ^= 1;
  }
  __syncthreads();
}

// Where element e goes in its finished range: stable by key.
template <int CAP, int NT>
__device__ __forceinline__ uint32_t final_slot(const SortSmem<CAP, NT> &S, uint32_t e) {
  const uint32_t f = S.P[e], l = S.Q[e];
  const float k = S.key[e];
  uint32_t pos = f;
  for (uint32_t j = f; j < l; j++) {
    const float kj = S.key[j];
    if (kj < k || (!(k < kj) && j < e)) pos++;
  }
  return pos;
}

template <int CAP, int NT>
__device__ __forceinline__ SortSmem<CAP, NT> &sort_smem() {
  extern __shared__ __align__(16) unsigned char s_sort[];
  return *reinterpret_cast<SortSmem<CAP, NT> *>(s_sort);
}

// Sorts the `len` loaded elements as one range and writes the indices to out.
template <int CAP, int NT>
__device__ __forceinline__ void sort_loaded(SortSmem<CAP, NT> &S, uint32_t len, uint32_t d, uint32_t *out,
                                            uint32_t *err) {
  if (threadIdx.x == 0) S.count[0] = S.big_count[0] = 0;
  __syncthreads();
  if (threadIdx.x < 32) push_range(S, 0, 0u, len, d, threadIdx.x, err);
  block_sort(S, err);
  for (uint32_t e = threadIdx.x; e < len; e += NT) out[final_slot(S, e)] = S.idx[e];
}

// One CTA per node of a level of nodes of at most CAP triangles.
template <int CAP, int NT>
__global__ void __launch_bounds__(NT) k_sort_segs(const rt_triangle *__restrict__ tris,
                                                  const uint8_t *__restrict__ axes, uint32_t n, uint32_t level,
                                                  uint32_t *idx, uint32_t *err) {
  SortSmem<CAP, NT> &S = sort_smem<CAP, NT>();
  const Item it = item_below(root_item(n), level, blockIdx.x);
  const uint32_t len = min(it.n, (uint32_t)CAP);
  const int axis = axes[it.rank];
  for (uint32_t e = threadIdx.x; e < len; e += NT) {
    const uint32_t o = level == 0 ? e : idx[it.off + e];
    S.idx[e] = o;
    S.key[e] = tri_key(tris[o], axis);
  }
  sort_loaded(S, len, 2u * (uint32_t)sortemu::floor_log2(it.n), idx + it.off, err);
}

// The ranges a big level left, one CTA each. A larger one has no depth left:
// introsort heap-sorts it, here one thread in global memory.
template <int CAP, int NT>
__global__ void __launch_bounds__(NT) k_sort_queue(float *key, uint32_t *idx,
                                                   const Range *__restrict__ queue, const uint32_t *qcount,
                                                   uint32_t *qhead, uint32_t *err) {
  SortSmem<CAP, NT> &S = sort_smem<CAP, NT>();
  __shared__ uint32_t s_item;
  const uint32_t count = *qcount;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(qhead, 1u);
    __syncthreads();
    if (s_item >= count) return;
    const Range r = queue[s_item];
    const uint32_t len = r.l - r.f;
    if (len > (uint32_t)CAP) {
      if (threadIdx.x == 0) sortemu::heap_sort(key + r.f, idx + r.f, (long)len);
      continue;
    }
    for (uint32_t e = threadIdx.x; e < len; e += NT) {
      S.key[e] = key[r.f + e];
      S.idx[e] = idx[r.f + e];
    }
    sort_loaded(S, len, r.d, idx + r.f, err);
  }
}

__device__ __forceinline__ rt_bvh_node leaf_node(const rt_triangle &t, uint32_t object) {
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
  nd.object = (int32_t)object;
  nd._pad1[0] = nd._pad1[1] = 0;
  return nd;
}

// The inner node of `it` from its children's records.
__device__ __forceinline__ void write_inner(rt_bvh_node *nodes, const Item &it) {
  const uint32_t k = it.rank - it.leaves, L = 2 * k + 1, R = 2 * k + 2;
  const rt_bvh_node a = nodes[L], b = nodes[R];
  rt_bvh_node nd;
  for (int c = 0; c < 3; c++) {
    nd.min[c] = (b.min[c] < a.min[c]) ? b.min[c] : a.min[c];
    nd.max[c] = (a.max[c] < b.max[c]) ? b.max[c] : a.max[c];
  }
  nd._pad0 = 0.0f;
  nd.left = (int32_t)L;
  nd.right = (int32_t)R;
  nd.object = -1;
  nd._pad1[0] = nd._pad1[1] = 0;
  nodes[it.node] = nd;
}

// One CTA per node of `level` (at most kTreeCap triangles): sorts that node
// and all below it, then writes their records.
template <int NT>
__global__ void __launch_bounds__(NT) k_subtrees(const rt_triangle *__restrict__ tris,
                                                 const uint8_t *__restrict__ axes, uint32_t n, uint32_t level,
                                                 const uint32_t *__restrict__ idx, rt_bvh_node *nodes, uint32_t *err,
                                                 int test_error_level) {
  constexpr int PER = (int)kTreeCap / NT;
  SortSmem<(int)kTreeCap, NT> &S = sort_smem<(int)kTreeCap, NT>();
  const Item top = item_below(root_item(n), level, blockIdx.x);
  // Slices below are local: offset 0 is the subtree's first triangle.
  Item root = top;
  root.off = 0;
  const uint32_t len = min(top.n, kTreeCap);
  for (uint32_t e = threadIdx.x; e < len; e += NT) S.idx[e] = level == 0 ? e : idx[top.off + e];
  uint32_t below = 0;
  for (; level_max(len, below) >= 2; below++) {
    __syncthreads();
    if (threadIdx.x == 0) {
      S.count[0] = S.big_count[0] = 0;
      if (blockIdx.x == 0 && (int)(level + below) == test_error_level) atomicOr(err, KERR_STACK_OVERFLOW);
    }
    __syncthreads();
    // Nodes above kInsertion are listed; the elements of the others are marked.
    if (level_max(len, below) > kInsertion)
      for (uint32_t i = threadIdx.x; i < (1u << below); i += NT) {
        const Item it = item_below(root, below, i);
        if (it.n > kInsertion) {
          const uint32_t k = atomicAdd(&S.count[0], 1u);  // disjoint ranges above kInsertion: fewer than kTreeCap / 16
          S.list[0][k] = it.off | ((it.off + it.n) << 16);
          S.depth[0][k] = (uint8_t)(2 * sortemu::floor_log2(it.n));
        }
      }
    for (uint32_t e = threadIdx.x; e < len; e += NT) {
      const Item it = item_holding(root, below, e);
      S.key[e] = tri_key(tris[S.idx[e]], axes[it.rank]);
      if (it.n <= kInsertion) {
        S.P[e] = (uint16_t)it.off;
        S.Q[e] = (uint16_t)(it.off + it.n);
      }
    }
    block_sort(S, err);
    uint32_t slot[PER], val[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const uint32_t e = threadIdx.x + j * NT;
      slot[j] = e < len ? final_slot(S, e) : 0u;
      val[j] = e < len ? S.idx[e] : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; j++)
      if (threadIdx.x + j * NT < len) S.idx[slot[j]] = val[j];
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < len; e += NT) {
    Item it = root;
    while (it.n > 1) it = child_item(it, e >= it.off + it.n / 2);
    const uint32_t o = S.idx[e];
    nodes[it.node] = leaf_node(tris[o], o);
  }
  for (int b = (int)below - 1; b >= 0; b--) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < (1u << b); i += NT) {
      const Item it = item_below(root, (uint32_t)b, i);
      if (it.n >= 2) write_inner(nodes, it);
    }
  }
}

// The inner nodes above `level`, by one CTA.
__global__ void __launch_bounds__(1024) k_top(uint32_t n, uint32_t level, rt_bvh_node *nodes) {
  for (int L = (int)level - 1; L >= 0; L--) {
    for (uint32_t i = threadIdx.x; i < (1u << L); i += 1024) write_inner(nodes, item_below(root_item(n), (uint32_t)L, i));
    __syncthreads();
  }
}

// --------------------------------------------------------------- big levels
// Device words of a build: queue count and head, barrier, error bits, and the
// range and tile counts of the two range lists.
enum : uint32_t { kCtrQueue = 0, kCtrHead = 1, kCtrErr = 2, kCtrBarrier = 3, kCtrRanges = 4, kCtrTiles = 6, kCtrWords = 16 };

struct BigLists {
  BigRange *ranges[2];
  uint32_t *tile_range[2];  // range of each tile
  uint2 *tile_count;        // !(x < p) and !(p < x) in each tile
  uint32_t max_ranges, max_tiles;
};

// A range of a big level, added by one CTA: to the queue when one CTA can
// finish it (or its depth limit has run out), else to the next round's
// ranges and their tiles.
__device__ __forceinline__ void push_big(const BigLists &B, int next, uint32_t f, uint32_t l, uint32_t d,
                                         Range *queue, uint32_t *ctr) {
  __shared__ uint32_t s_range, s_tile;
  const uint32_t n = l - f;
  if (n < 2) return;
  if (n <= kRangeCap || d == 0) {
    if (threadIdx.x == 0) queue[atomicAdd(ctr + kCtrQueue, 1u)] = Range{f, l, d};
    return;
  }
  const uint32_t tiles = (n + kTile - 1) / kTile;
  __syncthreads();
  if (threadIdx.x == 0) {
    s_range = atomicAdd(ctr + kCtrRanges + next, 1u);
    s_tile = atomicAdd(ctr + kCtrTiles + next, tiles);
    if (s_range >= B.max_ranges || s_tile + tiles > B.max_tiles) {
      atomicOr(ctr + kCtrErr, KERR_STACK_OVERFLOW);
      s_range = 0xffffffffu;
    } else {
      B.ranges[next][s_range] = BigRange{f, l, d, s_tile, 0u, 0u};
    }
  }
  __syncthreads();
  if (s_range != 0xffffffffu)
    for (uint32_t t = threadIdx.x; t < tiles; t += blockDim.x) B.tile_range[next][s_tile + t] = s_range;
}

// One level of nodes above kSegCap: keys, then introsort partition rounds
// over every range of the level at once, until each range is in the queue.
// A round has four phases, a grid barrier apart: the median of each range to
// its front; per tile the counts of !(x < p) and !(p < x); their rank lists P
// and Q; the search for K, the swaps and the two children. One CTA took the
// top levels before this (a CTA per node): 32.5 ms of a 1.31M-triangle build.
__global__ void __launch_bounds__(kBigThreads) k_big_level(const rt_triangle *__restrict__ tris,
                                                           const uint8_t *__restrict__ axes, uint32_t n,
                                                           uint32_t level, float *key, uint32_t *idx, uint32_t *P,
                                                           uint32_t *Q, BigLists B, Range *queue, uint32_t *ctr) {
  __shared__ uint32_t s_ge[kBigThreads / 32], s_le[kBigThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr uint32_t NW = kBigThreads / 32;
  uint32_t *err = ctr + kCtrErr;
  uint32_t target = 0;
  for (uint32_t e = blockIdx.x * kBigThreads + tid; e < n; e += gridDim.x * kBigThreads) {
    const Item it = item_holding(root_item(n), level, e);
    const uint32_t o = level == 0 ? e : __ldcg(idx + e);
    if (level == 0) idx[e] = o;
    key[e] = tri_key(tris[o], axes[it.rank]);
  }
  for (uint32_t i = blockIdx.x; i < (1u << level); i += gridDim.x) {
    const Item it = item_below(root_item(n), level, i);
    push_big(B, 0, it.off, it.off + it.n, 2u * (uint32_t)sortemu::floor_log2(it.n), queue, ctr);
  }
  if (!grid_barrier(ctr + kCtrBarrier, err, target)) return;
  for (int round = 0, cur = 0; round < kMaxRounds; round++, cur ^= 1) {
    // Lists written before the barrier: read past L1.
    const uint32_t nr = min(__ldcg(ctr + kCtrRanges + cur), B.max_ranges);
    const uint32_t nt = min(__ldcg(ctr + kCtrTiles + cur), B.max_tiles);
    if (nr == 0) return;
    BigRange *ranges = B.ranges[cur];
    for (uint32_t r = blockIdx.x * kBigThreads + tid; r < nr; r += gridDim.x * kBigThreads) {
      const uint32_t f = __ldcg(&ranges[r].f), l = __ldcg(&ranges[r].l);
      const uint32_t mid = f + (l - f) / 2;
      const float kf = __ldcg(key + f), ka = __ldcg(key + f + 1), kb = __ldcg(key + mid), kc = __ldcg(key + l - 1);
      const uint32_t m = median_of(ka, kb, kc, f + 1, mid, l - 1);
      const uint32_t vf = __ldcg(idx + f), vm = __ldcg(idx + m);
      key[f] = m == mid ? kb : (m == f + 1 ? ka : kc);
      idx[f] = vm;
      key[m] = kf;
      idx[m] = vf;
    }
    if (blockIdx.x == 0 && tid == 0) ctr[kCtrRanges + (cur ^ 1)] = ctr[kCtrTiles + (cur ^ 1)] = 0u;
    if (!grid_barrier(ctr + kCtrBarrier, err, target)) return;
    // Counts per tile.
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
      const BigRange &R = ranges[__ldcg(B.tile_range[cur] + t)];
      const uint32_t f = __ldcg(&R.f), l = __ldcg(&R.l), t0 = __ldcg(&R.tile0);
      const float pk = __ldcg(key + f);
      const uint32_t beg = f + 1 + (t - t0) * kTile, end = min(l, beg + kTile);
      uint32_t ge = 0, le = 0;
      for (uint32_t i = beg + tid; i < end; i += kBigThreads) {
        const float k = __ldcg(key + i);
        ge += !(k < pk);
        le += !(pk < k);
      }
      ge = __reduce_add_sync(0xffffffffu, ge);
      le = __reduce_add_sync(0xffffffffu, le);
      if (lane == 0) s_ge[warp] = ge, s_le[warp] = le;
      __syncthreads();
      if (warp == 0) {
        ge = __reduce_add_sync(0xffffffffu, lane < NW ? s_ge[lane] : 0u);
        le = __reduce_add_sync(0xffffffffu, lane < NW ? s_le[lane] : 0u);
        if (lane == 0) B.tile_count[t] = make_uint2(ge, le);
      }
      __syncthreads();
    }
    if (!grid_barrier(ctr + kCtrBarrier, err, target)) return;
    // Rank lists, both from the left.
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
      BigRange &R = ranges[__ldcg(B.tile_range[cur] + t)];
      const uint32_t f = __ldcg(&R.f), l = __ldcg(&R.l), t0 = __ldcg(&R.tile0);
      const float pk = __ldcg(key + f);
      uint32_t ge = 0, le = 0;
      for (uint32_t u = t0 + tid; u < t; u += kBigThreads) {
        const uint2 c = __ldcg(B.tile_count + u);
        ge += c.x;
        le += c.y;
      }
      ge = __reduce_add_sync(0xffffffffu, ge);
      le = __reduce_add_sync(0xffffffffu, le);
      if (lane == 0) s_ge[warp] = ge, s_le[warp] = le;
      __syncthreads();
      ge = __reduce_add_sync(0xffffffffu, lane < NW ? s_ge[lane] : 0u);
      le = __reduce_add_sync(0xffffffffu, lane < NW ? s_le[lane] : 0u);
      __syncthreads();
      const uint32_t beg = f + 1 + (t - t0) * kTile, end = min(l, beg + kTile);
      // Warp w takes the w-th run of the tile, in order.
      constexpr uint32_t RUN = kTile / NW;
      const uint32_t wb = min(end, beg + warp * RUN), we = min(end, wb + RUN);
      float k[RUN / 32];
      uint32_t wg = 0, wl = 0;
#pragma unroll
      for (uint32_t j = 0; j < RUN / 32; j++) {
        const uint32_t i = wb + j * 32 + lane;
        k[j] = i < we ? __ldcg(key + i) : 0.0f;
        wg += __popc(__ballot_sync(0xffffffffu, i < we && !(k[j] < pk)));
        wl += __popc(__ballot_sync(0xffffffffu, i < we && !(pk < k[j])));
      }
      if (lane == 0) s_ge[warp] = wg, s_le[warp] = wl;
      __syncthreads();
      ge += __reduce_add_sync(0xffffffffu, lane < warp ? s_ge[lane] : 0u);
      le += __reduce_add_sync(0xffffffffu, lane < warp ? s_le[lane] : 0u);
      const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
      for (uint32_t j = 0; j < RUN / 32; j++) {
        const uint32_t i = wb + j * 32 + lane;
        const bool g = i < we && !(k[j] < pk), q = i < we && !(pk < k[j]);
        const uint32_t bg = __ballot_sync(0xffffffffu, g), bq = __ballot_sync(0xffffffffu, q);
        if (g) P[f + ge + __popc(bg & lt)] = i;
        if (q) Q[f + le + __popc(bq & lt)] = i;
        ge += __popc(bg);
        le += __popc(bq);
      }
      // The last warp of the last tile ends on the range's totals.
      if (end == l && warp == NW - 1 && lane == 0) R.ge = ge, R.le = le;
      __syncthreads();
    }
    if (!grid_barrier(ctr + kCtrBarrier, err, target)) return;
    // K, the swaps (shared out over the range's tiles) and the children.
    for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
      const BigRange &R = ranges[__ldcg(B.tile_range[cur] + t)];
      const uint32_t f = __ldcg(&R.f), l = __ldcg(&R.l), d = __ldcg(&R.d), t0 = __ldcg(&R.tile0);
      const uint32_t ge = __ldcg(&R.ge), le = __ldcg(&R.le);
      uint32_t lo = 0, hi = min(ge, le);
      while (lo < hi) {
        const uint32_t step = (hi - lo + kBigThreads - 1) / kBigThreads;
        const uint32_t j = lo + (tid + 1) * step - 1;
        const uint32_t c =
            (uint32_t)__syncthreads_count(j < hi && __ldcg(P + f + j) < __ldcg(Q + f + le - 1 - j) ? 1 : 0);
        lo += c * step;
        hi = min(hi, lo + step - 1);
      }
      const uint32_t K = lo, tiles = (l - f + kTile - 1) / kTile;
      const uint32_t share = (K + tiles - 1) / tiles, j1 = min(K, (t - t0 + 1) * share);
      for (uint32_t j = (t - t0) * share + tid; j < j1; j += kBigThreads) {
        const uint32_t a = __ldcg(P + f + j), b = __ldcg(Q + f + le - 1 - j);
        const float ka = __ldcg(key + a), kb = __ldcg(key + b);
        const uint32_t va = __ldcg(idx + a), vb = __ldcg(idx + b);
        key[a] = kb;
        idx[a] = vb;
        key[b] = ka;
        idx[b] = va;
      }
      if (t == t0) {
        uint32_t cut = K < ge ? __ldcg(P + f + K) : 0xffffffffu;
        if (K >= 1) cut = min(cut, __ldcg(Q + f + le - K));
        if (cut <= f || cut >= l) {  // cannot happen for finite keys
          if (tid == 0) atomicOr(err, KERR_BAD_INDEX);
        } else {
          push_big(B, cur ^ 1, f, cut, d - 1, queue, ctr);
          push_big(B, cur ^ 1, cut, l, d - 1, queue, ctr);
        }
      }
    }
    if (!grid_barrier(ctr + kCtrBarrier, err, target)) return;
  }
}

// --------------------------------------------------------------------- host
constexpr size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

// Scratch of a build of n triangles, carved from one area.
struct BuildScratch {
  float *key;
  uint32_t *idx, *P, *Q, *ctr;
  Range *queue;
  uint8_t *axes;
  BigLists big;
};
constexpr uint32_t big_ranges(uint32_t n) { return n / kRangeCap + 1; }
constexpr uint32_t big_tiles(uint32_t n) { return n / kTile + big_ranges(n) + 1; }
constexpr size_t build_scratch_bytes(uint32_t n) {
  return 256 + 4 * align_up(4ull * n) + align_up(sizeof(Range) * (size_t)n) + align_up(2ull * n) +
         2 * align_up(sizeof(BigRange) * (size_t)big_ranges(n)) + 2 * align_up(4ull * big_tiles(n)) +
         align_up(8ull * big_tiles(n));
}
BuildScratch carve_build(unsigned char *p, uint32_t n) {
  auto take = [&p](size_t bytes) {
    unsigned char *q = p;
    p += align_up(bytes);
    return q;
  };
  BuildScratch s;
  s.ctr = (uint32_t *)take(256);
  s.key = (float *)take(4ull * n);
  s.idx = (uint32_t *)take(4ull * n);
  s.P = (uint32_t *)take(4ull * n);
  s.Q = (uint32_t *)take(4ull * n);
  s.queue = (Range *)take(sizeof(Range) * (size_t)n);
  s.axes = (uint8_t *)take(2ull * n);
  s.big.max_ranges = big_ranges(n);
  s.big.max_tiles = big_tiles(n);
  for (int i = 0; i < 2; i++) s.big.ranges[i] = (BigRange *)take(sizeof(BigRange) * (size_t)s.big.max_ranges);
  for (int i = 0; i < 2; i++) s.big.tile_range[i] = (uint32_t *)take(4ull * s.big.max_tiles);
  s.big.tile_count = (uint2 *)take(8ull * s.big.max_tiles);
  return s;
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int CAP, int NT>
cudaError_t launch_segs(const rt_triangle *tris, const BuildScratch &s, uint32_t n, uint32_t level, cudaStream_t st) {
  auto kern = k_sort_segs<CAP, NT>;
  cudaError_t e = allow_smem(kern, sizeof(SortSmem<CAP, NT>));
  if (e != cudaSuccess) return e;
  kern<<<1u << level, NT, sizeof(SortSmem<CAP, NT>), st>>>(tris, s.axes, n, level, s.idx, s.ctr + kCtrErr);
  return cudaGetLastError();
}

// Levels of the tree of n triangles, the leaves' included.
uint32_t tree_levels(uint32_t n) {
  const uint32_t d = (uint32_t)sortemu::floor_log2(n);
  return (n & (n - 1)) ? d + 2 : d + 1;
}

// Enqueues the draws.
cudaError_t enqueue_axes(uint32_t seed, uint32_t n, const BuildScratch &s, cudaStream_t st) {
  const uint64_t count = 2ull * n - 1, runs = (count + kAxisRun - 1) / kAxisRun;
  k_axes<<<(uint32_t)((runs + kAxisWarps - 1) / kAxisWarps), 32 * kAxisWarps, 0, st>>>(glibc_axis_jump(seed), count,
                                                                                       s.axes);
  return cudaGetLastError();
}

// Enqueues the build of d_nodes; s.axes holds the draws and s.ctr is zero.
// The node size of a level picks its kernel: up to kTreeCap a CTA of 256
// takes the whole subtree (1,024 CTAs at 1.31M triangles), up to kSegCap one
// CTA still holds a node in shared memory; above, the grid works together.
cudaError_t enqueue_build(const rt_triangle *d_tris, uint32_t n, const BuildScratch &s, rt_bvh_node *d_nodes,
                          int test_error_level, cudaStream_t st) {
  int dev = 0, sms = 0, per_sm = 0, per_sm_q = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  auto kq = k_sort_queue<(int)kRangeCap, 1024>;
  using QSmem = SortSmem<(int)kRangeCap, 1024>;
  uint32_t level = 0;
  for (; level_max(n, level) > kTreeCap && e == cudaSuccess; level++) {
    const uint32_t most = level_max(n, level);
    if (most > kSegCap) {
      if (per_sm == 0) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_big_level, kBigThreads, 0);
        if (e == cudaSuccess) e = allow_smem(kq, sizeof(QSmem));
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_q, kq, 1024, sizeof(QSmem));
        per_sm = std::max(1, std::min(per_sm, 2));
        per_sm_q = std::max(1, per_sm_q);
      }
      if (e == cudaSuccess) e = cudaMemsetAsync(s.ctr, 0, 4 * kCtrErr, st);
      if (e == cudaSuccess)
        e = cudaMemsetAsync(s.ctr + kCtrBarrier, 0, 4 * (kCtrWords - kCtrBarrier), st);
      if (e != cudaSuccess) return e;
      const uint32_t want = (n + kTile - 1) / kTile;
      const uint32_t grid = std::min<uint32_t>((uint32_t)(sms * per_sm), want);
      uint32_t nn = n, lv = level;
      const uint8_t *axes = s.axes;
      float *key = s.key;
      uint32_t *idx = s.idx, *P = s.P, *Q = s.Q, *ctr = s.ctr;
      BigLists big = s.big;
      Range *queue = s.queue;
      void *args[] = {&d_tris, &axes, &nn, &lv, &key, &idx, &P, &Q, &big, &queue, &ctr};
      e = cudaLaunchCooperativeKernel((const void *)k_big_level, dim3(grid), dim3(kBigThreads), args, 0, st);
      if (e != cudaSuccess) return e;
      kq<<<sms * per_sm_q, 1024, sizeof(QSmem), st>>>(s.key, s.idx, s.queue, s.ctr + kCtrQueue, s.ctr + kCtrHead,
                                                      s.ctr + kCtrErr);
      e = cudaGetLastError();
    } else if (most > 8192) {
      e = launch_segs<(int)kSegCap, 1024>(d_tris, s, n, level, st);
    } else if (most > 4096) {
      e = launch_segs<8192, 1024>(d_tris, s, n, level, st);
    } else {
      e = launch_segs<4096, 512>(d_tris, s, n, level, st);
    }
    if (e == cudaSuccess && (int)level == test_error_level) {
      k_flag_error<<<1, 1, 0, st>>>(s.ctr + kCtrErr, KERR_STACK_OVERFLOW);
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) return e;
  auto kt = k_subtrees<256>;
  using TSmem = SortSmem<(int)kTreeCap, 256>;
  if ((e = allow_smem(kt, sizeof(TSmem))) != cudaSuccess) return e;
  kt<<<1u << level, 256, sizeof(TSmem), st>>>(d_tris, s.axes, n, level, s.idx, d_nodes, s.ctr + kCtrErr,
                                              test_error_level);
  if (level > 0) k_top<<<1, 1024, 0, st>>>(n, level, d_nodes);
  return cudaGetLastError();
}

#define BUILD_CHECK(x)                                                                       \
  do {                                                                                       \
    cudaError_t e_ = (x);                                                                    \
    if (e_ != cudaSuccess) {                                                                 \
      std::snprintf(errbuf, errlen, "bvh build: %s (%s:%d)", cudaGetErrorString(e_), __FILE__, \
                    __LINE__);                                                               \
      status = RT_ERR_CUDA;                                                                  \
      goto done;                                                                             \
    }                                                                                        \
  } while (0)

}  // namespace

rt_status gpu_build_bvh(const rt_triangle *d_tris, uint32_t n, uint32_t bvh_seed, rt_bvh_node *d_nodes,
                        ScratchPool &pool, cudaStream_t st, float *ms_out, uint32_t *depth_out, char *errbuf,
                        size_t errlen, int test_error_level) {
  rt_status status = RT_SUCCESS;
  unsigned char *mem = nullptr;
  BuildScratch s;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  BUILD_CHECK(cudaEventCreate(&e0));
  BUILD_CHECK(cudaEventCreate(&e1));
  BUILD_CHECK(scratch_alloc((void **)&mem, build_scratch_bytes(n), pool, st));
  s = carve_build(mem, n);
  BUILD_CHECK(cudaEventRecord(e0, st));
  BUILD_CHECK(enqueue_axes(bvh_seed, n, s, st));
  BUILD_CHECK(cudaMemsetAsync(s.ctr, 0, 4 * kCtrWords, st));
  BUILD_CHECK(enqueue_build(d_tris, n, s, d_nodes, test_error_level, st));
  BUILD_CHECK(cudaEventRecord(e1, st));
  {
    uint32_t bits = 0;
    BUILD_CHECK(cudaMemcpyAsync(&bits, s.ctr + kCtrErr, sizeof(bits), cudaMemcpyDeviceToHost, st));
    BUILD_CHECK(cudaStreamSynchronize(st));
    if (bits != 0) {
      std::snprintf(errbuf, errlen, "bvh build: internal sort error (bits 0x%x)", bits);
      status = RT_ERR_INTERNAL;
    }
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms_out) *ms_out = ms;
    if (depth_out) *depth_out = tree_levels(n);
  }
done:
  if (mem) cudaFreeAsync(mem, st);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  return status;
}

}  // namespace rtgb

// ---------------------------------------------------------------------------
// Allocation-free build: rtBuildBvhNoAlloc.
//
// For callers that cannot allocate device memory, the same kernels run on a
// fixed scratch area that is part of the library image: a file-scope
// __device__ array sized for kNoAllocMaxTriangles triangles (about 2 MB,
// held by every GPU that loads the library until the process exits). The
// host keeps one static word, so a call performs no allocation of any kind.
// All calls share both: calls must not
// overlap (they are serialised on the host by a mutex and each call waits
// for its own GPU work before returning; calls issued by other means on the
// same device while one is running would race on the shared array).
#include <mutex>

namespace rtgb {
namespace {

constexpr uint32_t kNoAllocMaxTriangles = 65536;

static __device__ __align__(256) unsigned char g_noalloc_scratch[build_scratch_bytes(kNoAllocMaxTriangles)];

static uint32_t g_na_bits;  // the error word, read back
static std::mutex g_na_mu;
constexpr int kNaMaxDevices = 64;
static unsigned char *g_na_dev[kNaMaxDevices];  // device address of the scratch array, per device

}  // namespace
}  // namespace rtgb

extern "C" rt_status rtBuildBvhNoAlloc(const rt_triangle *d_triangles, uint32_t n, uint32_t bvh_seed,
                                       rt_bvh_node *d_nodes, void *stream) {
  using namespace rtgb;
  if (!d_triangles || !d_nodes || n == 0 || n > kNoAllocMaxTriangles) return RT_ERR_INVALID_ARGUMENT;
  if ((uintptr_t)d_triangles % 16 || (uintptr_t)d_nodes % 16) return RT_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> guard(g_na_mu);
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDevices) return RT_ERR_CUDA;
  if (!g_na_dev[dev]) {
    // Once per device, with that device current: host code cannot use the
    // array's name as a device address, so look the address up.
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return RT_ERR_CUDA;
    g_na_dev[dev] = static_cast<unsigned char *>(p);
  }
  const BuildScratch s = carve_build(g_na_dev[dev], n);
  // From the first enqueue on, every return waits for the work already
  // queued on `st`: the next call (under the same lock, possibly on another
  // stream) reuses the scratch array.
  auto drain = [st](rt_status r) {
    cudaStreamSynchronize(st);
    return r;
  };
  constexpr uint32_t kNonFinite = 0x100u;
  if (enqueue_axes(bvh_seed, n, s, st) != cudaSuccess) return drain(RT_ERR_CUDA);
  // The error word survives from earlier calls: clear it.
  if (cudaMemsetAsync(s.ctr, 0, 4 * kCtrWords, st) != cudaSuccess) return drain(RT_ERR_CUDA);
  // Non-finite vertices are rejected before any sort runs: the sort replay
  // assumes keys that IEEE `<` orders totally.
  k_check_finite<<<(n + 255) / 256, 256, 0, st>>>(d_triangles, n, s.ctr + kCtrErr, kNonFinite);
  if (cudaGetLastError() != cudaSuccess) return drain(RT_ERR_CUDA);
  if (cudaMemcpyAsync(&g_na_bits, s.ctr + kCtrErr, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return drain(RT_ERR_CUDA);
  if (cudaStreamSynchronize(st) != cudaSuccess) return RT_ERR_CUDA;
  if (g_na_bits & kNonFinite) return RT_ERR_INVALID_SCENE;
  if (enqueue_build(d_triangles, n, s, d_nodes, -1, st) != cudaSuccess) return drain(RT_ERR_CUDA);
  if (cudaMemcpyAsync(&g_na_bits, s.ctr + kCtrErr, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return drain(RT_ERR_CUDA);
  if (cudaStreamSynchronize(st) != cudaSuccess) return RT_ERR_CUDA;
  return g_na_bits ? RT_ERR_INTERNAL : RT_SUCCESS;
}
