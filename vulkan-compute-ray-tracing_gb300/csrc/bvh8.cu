// 8-wide traversal tree (bvh8) collapsed from the children-pair layout.
//
// The tree is the reference's (or the selected builder's) binary tree with
// levels folded together; no box is recomputed or moved. Each bvh8 node
// holds up to eight children. By default the binary nodes that become bvh8
// nodes are chosen by the surface area heuristic (the SAH collapse below,
// the dynamic program of Ylitie et al., "Efficient Incoherent Ray Traversal
// on GPUs Through Compressed Wide BVHs", HPG 2017, for single-triangle
// leaves). The alternative ("bvh8.collapse" 0) starts from one inner node's
// two children and replaces the inner child with the largest surface area
// by its own two children until there are eight or only leaves are left
// (greedy collapse as in Wald et al., "Getting Rid of Packets", RT 2008); a
// node with fewer than eight children then holds leaves only, which bounds
// the node count by (4n - 1) / 7 for n leaves, the capacity reserved.
//
// Slots are assigned by position (Ylitie et al.'s octant order): slot s,
// read as three bits (x, y, z), stands for the corner of the node on the
// positive side of the axes whose bit is set. Each child goes to the free
// slot whose corner direction best matches the offset of its box centre
// from the node's centre (greedy on the cost -sum_k sign_k(s) * offset_k,
// lowest cost first, ties to the lower child then the lower slot). A ray
// whose direction has sign bits o (bit k set when d_k < 0) then meets the
// children roughly in increasing order of s ^ o, so the traversal orders
// the children it enters with one XOR instead of sorting their distances.
//
// The fold is built in fp32 (8 slots of 32 bytes: (lo.x, lo.y, lo.z, hi.x),
// (hi.y, hi.z, ref, 0), empty slots ref INT_MIN) and then stored quantized,
// 96 bytes per node (k_quantize8, the compression of Ylitie et al. with
// explicit child refs):
//   words 0-2    origin o: the lo corner of the union of the children
//   word 3       int8 exponents ex, ey, ez; the mask of filled slots
//   words 4-15   8-bit child bounds qlo.x[8], qlo.y, qlo.z, qhi.x, qhi.y,
//                qhi.z (slot s in byte s & 3 of word 2 * plane + (s >> 2));
//                an empty slot has qlo = 255, qhi = 0
//   words 16-23  child refs; an empty slot holds ~0 (the leaf of tpre
//                record 0)
// A child's box decodes to o + q * 2^e per axis. qlo is rounded down and
// qhi up, and both are checked against the fp32 box, so the decoded box
// always contains the original one. Refs: >= 0 is an inner child (its node
// number); ~k is a leaf (tpre record k, as in bvh2). An empty slot's
// inverted box misses every ray whose 1/d is not flushed to zero on all
// three axes; should one still pass, its ref sends the lane to test record
// 0, a real triangle, which cannot change a closest hit. The traversal
// therefore needs no filled-mask test per slot.
// Nodes are numbered breadth first, level by level; the inner children of
// one node are consecutive, in slot order.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstring>

#include "grid_sync.cuh"
#include "rt_internal.h"

namespace rtgb {

// Quantizes one node: box[s] = (lo.xyz, hi.xyz) of the children in the
// slots of `fmask`, refs copied as given, into the 24 words of a bvh8 node
// (layout above). Per axis the origin is the children's union lo and the
// step the smallest power of two 2^e with extent <= 255 * 2^e; each bound
// becomes a byte, rounded down for lo and up for hi, then checked in fp64
// against the fp32 bound and moved outward if needed, so the decoded box
// o + q * 2^e always contains the original. Empty slots get qlo = 255,
// qhi = 0 and ref ~0. False when some box does not fit the grid (or fmask is
// empty).
__host__ __device__ inline bool quantize_node8(const float box[8][6], const int32_t ref[8], uint32_t fmask,
                                               uint32_t w[24]) {
  fmask &= 0xffu;
  bool ok = fmask != 0;
  if (!ok) fmask = 1;
  for (int i = 0; i < 24; i++) w[i] = 0;
  uint32_t ebytes = fmask << 24;
  for (int k = 0; k < 3; k++) {
    float ulo = 0.0f, uhi = 0.0f;
    bool first = true;
    for (int s = 0; s < 8; s++) {
      if (!((fmask >> s) & 1u)) continue;
      ulo = first ? box[s][k] : fminf(ulo, box[s][k]);
      uhi = first ? box[s][3 + k] : fmaxf(uhi, box[s][3 + k]);
      first = false;
    }
    const double E = (double)uhi - (double)ulo;
    int e = -126;
    if (E > 0.0) {
      int e0 = 0;
      frexp(E, &e0);  // 2^(e0 - 1) <= E < 2^e0, so 2^(e0 - 9) is too small a step
      e = (E <= 255.0 * ldexp(1.0, e0 - 8)) ? e0 - 8 : e0 - 7;
      e = e < -126 ? -126 : (e > 127 ? 127 : e);
    }
    // Steps are powers of two: multiplying by the inverse divides exactly.
    const double sc = ldexp(1.0, e), inv = ldexp(1.0, -e);
    if (E > 255.0 * sc) ok = false;
    for (int s = 0; s < 8; s++) {
      int ql = 255, qh = 0;
      if ((fmask >> s) & 1u) {
        const double lo = box[s][k], hi = box[s][3 + k];
        ql = (int)floor((lo - (double)ulo) * inv);
        ql = ql < 0 ? 0 : (ql > 255 ? 255 : ql);
        while ((double)ulo + ql * sc > lo) {
          if (ql == 0) {
            ok = false;
            break;
          }
          ql--;
        }
        qh = (int)ceil((hi - (double)ulo) * inv);
        qh = qh < 0 ? 0 : (qh > 255 ? 255 : qh);
        while ((double)ulo + qh * sc < hi) {
          if (qh == 255) {
            ok = false;
            break;
          }
          qh++;
        }
      }
      w[4 + 2 * k + (s >> 2)] |= (uint32_t)ql << (8 * (s & 3));
      w[10 + 2 * k + (s >> 2)] |= (uint32_t)qh << (8 * (s & 3));
    }
    union {
      float f;
      uint32_t u;
    } bits;
    bits.f = ulo;
    w[k] = bits.u;
    ebytes |= ((uint32_t)(e & 0xff)) << (8 * k);
  }
  w[3] = ebytes;
  for (int s = 0; s < 8; s++) w[16 + s] = (fmask >> s) & 1u ? (uint32_t)ref[s] : ~0u;
  return ok;
}

// Octant slot assignment (see the top of this file) of `cnt` child boxes
// (lo.xyz, hi.xyz): slot_of[i] receives child i's slot. Only additions and
// subtractions of the box coordinates are used (twice the centre offsets),
// so host and device give the same assignment.
__host__ __device__ inline void assign_octant_slots(const float (*box)[6], int cnt, int slot_of[8]) {
  float c2[3];
  for (int k = 0; k < 3; k++) {
    float ulo = box[0][k], uhi = box[0][3 + k];
    for (int i = 1; i < cnt; i++) {
      ulo = fminf(ulo, box[i][k]);
      uhi = fmaxf(uhi, box[i][3 + k]);
    }
    c2[k] = ulo + uhi;
  }
  float off[8][3];
  for (int i = 0; i < cnt; i++)
    for (int k = 0; k < 3; k++) off[i][k] = (box[i][k] + box[i][3 + k]) - c2[k];
  uint32_t used_slots = 0, used_kids = 0;
  for (int i = 0; i < 8; i++) slot_of[i] = -1;
  for (int round = 0; round < cnt; round++) {
    float best = 0.0f;
    int bi = -1, bs = -1;
    for (int i = 0; i < cnt; i++) {
      if ((used_kids >> i) & 1u) continue;
      for (int s = 0; s < 8; s++) {
        if ((used_slots >> s) & 1u) continue;
        float cost = 0.0f;
        for (int k = 0; k < 3; k++) cost = ((s >> k) & 1) ? cost - off[i][k] : cost + off[i][k];
        if (bi < 0 || cost < best) {
          best = cost;
          bi = i;
          bs = s;
        }
      }
    }
    slot_of[bi] = bs;
    used_kids |= 1u << bi;
    used_slots |= 1u << bs;
  }
}

namespace {

struct Slot {
  float lo[3], hi[3];
  int32_t ref;
};

__device__ __forceinline__ float slot_area(const Slot &s) {
  float dx = s.hi[0] - s.lo[0], dy = s.hi[1] - s.lo[1], dz = s.hi[2] - s.lo[2];
  return dx * dy + dy * dz + dz * dx;
}

// The two children of bvh2 pair p.
__device__ __forceinline__ void load_pair(const float4 *__restrict__ bvh2, int32_t p, Slot &c0, Slot &c1) {
  const float4 *N = bvh2 + 4ll * p;
  const float4 a = N[0], b = N[1], c = N[2], d = N[3];
  c0.lo[0] = a.x, c0.lo[1] = a.y, c0.hi[0] = a.z, c0.hi[1] = a.w, c0.lo[2] = b.x, c0.hi[2] = b.y;
  c1.lo[0] = c.x, c1.lo[1] = c.y, c1.hi[0] = c.z, c1.hi[1] = c.w, c1.lo[2] = d.x, c1.hi[2] = d.y;
  c0.ref = __float_as_int(b.z);
  c1.ref = __float_as_int(d.z);
}

// ---- SAH collapse: which bvh2 pairs become 8-wide nodes.
// A ray reaches an 8-wide node with probability proportional to the node's
// box area, and every leaf occupies one slot wherever it goes, so the fold
// that minimises the summed area of the chosen nodes minimises the expected
// node visits (the surface area heuristic with fixed leaf cost). Bottom-up
// over the pairs: D(p, j), j = 1..8, is the least summed area for covering
// pair p's subtree with at most j slots, either p itself as one slot (it
// becomes a node: C(p) = area(p) + the best split of 8 slots between its
// children) or its children splitting the j slots; a leaf costs 0. Each
// pair stores D(p, 1..8) and its choices: the split of j slots for j = 2..8
// (0: p stays one slot) and the split of 8 slots when p is a node.

// Parent pair of every inner pair and of every leaf (the root pair: -1).
__global__ void k_pair_parents(const float4 *__restrict__ bvh2, uint32_t n_pairs, int32_t *__restrict__ parent,
                               int32_t *__restrict__ leaf_parent, uint32_t ntris, uint32_t *__restrict__ err) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_pairs) return;
  const int32_t refs[2] = {__float_as_int(bvh2[4ull * p + 1].z), __float_as_int(bvh2[4ull * p + 3].z)};
  for (int c = 0; c < 2; c++) {
    const int32_t r = refs[c];
    if (r >= 0 ? (uint32_t)r >= n_pairs : (uint32_t)~r >= ntris) {
      atomicOr(err, 1u);
      continue;
    }
    if (r >= 0) parent[r] = (int32_t)p;
    else leaf_parent[~r] = (int32_t)p;
  }
}

// One thread per leaf climbs towards the root; the second thread to reach a
// pair (both children done) computes its costs and climbs on.
__global__ void k_collapse_costs(const float4 *__restrict__ bvh2, uint32_t n_pairs, uint32_t ntris,
                                 const int32_t *__restrict__ parent, const int32_t *__restrict__ leaf_parent,
                                 uint32_t *__restrict__ arrivals, float *__restrict__ cost,
                                 uint32_t *__restrict__ choice, uint32_t *__restrict__ err) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ntris) return;
  int32_t p = leaf_parent[k];
  for (int climb = 0; p >= 0; climb++) {
    if ((uint32_t)p >= n_pairs || climb > 128) {
      atomicOr(err, 1u);
      return;
    }
    if (atomicAdd(arrivals + p, 1u) == 0u) return;
    __threadfence();
    Slot c[2];
    load_pair(bvh2, p, c[0], c[1]);
    if ((c[0].ref >= 0 && (uint32_t)c[0].ref >= n_pairs) || (c[1].ref >= 0 && (uint32_t)c[1].ref >= n_pairs)) {
      atomicOr(err, 1u);
      return;
    }
    float dc[2][9];
    for (int i = 0; i < 2; i++)
      for (int j = 1; j <= 8; j++) dc[i][j] = c[i].ref >= 0 ? __ldcg(cost + 8ull * c[i].ref + (j - 1)) : 0.0f;
    Slot u = c[0];
    for (int a = 0; a < 3; a++) {
      u.lo[a] = fminf(c[0].lo[a], c[1].lo[a]);
      u.hi[a] = fmaxf(c[0].hi[a], c[1].hi[a]);
    }
    // Best split of j slots between the children, the lower left share first on ties.
    auto split = [&](int j, int &kbest) {
      float best = __int_as_float(0x7f800000);
      kbest = 1;
      for (int l = 1; l < j; l++) {
        const float v = dc[0][l] + dc[1][j - l];
        if (v < best) {
          best = v;
          kbest = l;
        }
      }
      return best;
    };
    int k8;
    const float as_node = slot_area(u) + split(8, k8);
    uint32_t ch = (uint32_t)k8 << 28;
    __stcg(cost + 8ull * p, as_node);
    for (int j = 2; j <= 8; j++) {
      int kj;
      const float v = split(j, kj);
      const bool keep = as_node <= v;
      __stcg(cost + 8ull * p + (j - 1), keep ? as_node : v);
      if (!keep) ch |= (uint32_t)kj << (4 * (j - 2));
    }
    __stcg(choice + p, ch);
    __threadfence();
    p = parent[p];
  }
}

// The SAH choices expanded: pair p0's slots as a node.
__device__ __forceinline__ int sah_slots(const float4 *__restrict__ bvh2, uint32_t n_pairs,
                                         const uint32_t *__restrict__ choice, int32_t p0, Slot (&S)[8],
                                         uint32_t *__restrict__ err) {
  struct Item {
    Slot s;
    int j;
  };
  Item st[8];
  int sp = 0, cnt = 0;
  Slot c0, c1;
  load_pair(bvh2, p0, c0, c1);
  const int k8 = (int)(__ldg(choice + p0) >> 28);
  if (k8 < 1 || k8 > 7) {
    atomicOr(err, 1u);
    return 0;
  }
  st[sp++] = Item{c1, 8 - k8};
  st[sp++] = Item{c0, k8};
  while (sp > 0) {
    const Item it = st[--sp];
    int kj = 0;
    if (it.s.ref >= 0 && it.j >= 2) {
      if ((uint32_t)it.s.ref >= n_pairs) {
        atomicOr(err, 1u);
        return 0;
      }
      kj = (int)((__ldg(choice + it.s.ref) >> (4 * (it.j - 2))) & 15u);
    }
    if (kj == 0) {
      if (cnt >= 8) {
        atomicOr(err, 1u);
        return 0;
      }
      S[cnt++] = it.s;
      continue;
    }
    if (kj >= it.j || sp + 2 > 8) {
      atomicOr(err, 1u);
      return 0;
    }
    load_pair(bvh2, it.s.ref, c0, c1);
    st[sp++] = Item{c1, it.j - kj};
    st[sp++] = Item{c0, kj};
  }
  return cnt;
}

// One frontier node: bvh2 pair p0 expanded into the 8 slots at `o`. Returns
// its number of inner children.
__device__ __forceinline__ uint32_t expand_node(const float4 *__restrict__ bvh2, uint32_t n_pairs, int32_t p0,
                                                float4 *__restrict__ o, const uint32_t *__restrict__ choice,
                                                uint32_t *__restrict__ err) {
  Slot S[8];
  int cnt = 0;
  if (p0 < 0 || (uint32_t)p0 >= n_pairs) {
    atomicOr(err, 1u);
  } else if (choice) {
    cnt = sah_slots(bvh2, n_pairs, choice, p0, S, err);
  } else {
    load_pair(bvh2, p0, S[0], S[1]);
    cnt = 2;
    while (cnt < 8) {
      int pick = -1;
      float best = -1.0f;
      for (int i = 0; i < cnt; i++) {
        if (S[i].ref < 0) continue;
        const float a = slot_area(S[i]);
        if (a > best) {
          best = a;
          pick = i;
        }
      }
      if (pick < 0) break;
      const int32_t p = S[pick].ref;
      if ((uint32_t)p >= n_pairs) {
        atomicOr(err, 1u);
        break;
      }
      load_pair(bvh2, p, S[pick], S[cnt]);
      cnt++;
    }
  }
  const float inf = __int_as_float(0x7f800000);
  for (int s = 0; s < 8; s++) {
    o[2 * s] = make_float4(inf, inf, inf, inf);
    o[2 * s + 1] = make_float4(inf, inf, __int_as_float(INT_MIN), 0.0f);
  }
  uint32_t inner = 0;
  if (cnt > 0) {
    float box[8][6];
    for (int i = 0; i < cnt; i++)
      for (int k = 0; k < 3; k++) {
        box[i][k] = S[i].lo[k];
        box[i][3 + k] = S[i].hi[k];
      }
    int slot_of[8];
    assign_octant_slots(box, cnt, slot_of);
    for (int i = 0; i < cnt; i++) {
      const int s = slot_of[i];
      o[2 * s] = make_float4(S[i].lo[0], S[i].lo[1], S[i].lo[2], S[i].hi[0]);
      o[2 * s + 1] = make_float4(S[i].hi[1], S[i].hi[2], __int_as_float(S[i].ref), 0.0f);
      inner += S[i].ref >= 0 ? 1u : 0u;
    }
  }
  return inner;
}

constexpr int kFoldThreads = 128;
constexpr uint32_t kFoldWarps = kFoldThreads / 32;
// Device words of a fold: barrier counter, error bits (1, 2 bad reference, 4
// capacity, 8 box off its grid, KERR_TIMEOUT << 4), nodes, levels.
enum : uint32_t { kFoldBarrier = 0, kFoldErr = 1, kFoldNodes = 2, kFoldLevels = 3, kFoldWords = 8 };
constexpr uint32_t kFoldTimeout = KERR_TIMEOUT << 4;

// The whole fold, level by level, in one cooperative launch: node base + f of
// a level is pair frontier[f]; its inner children are numbered after the
// level, in order, and are the next frontier. Each CTA keeps to one run of
// the frontier: it expands its nodes and counts their inner children, then
// (after a barrier) knows the counts before it and numbers them. 13 levels of
// 1.31M triangles in 0.55 ms (1.6 with three launches and a host round trip a
// level), 12,012 triangles in 0.2 (0.6).
__global__ void __launch_bounds__(kFoldThreads) k_fold8(const float4 *__restrict__ bvh2, uint32_t n_pairs,
                                                        const uint32_t *__restrict__ choice, float4 *bvh8,
                                                        uint32_t cap, int32_t *fr0, int32_t *fr1, uint32_t *inner_cnt,
                                                        uint32_t *counts, uint32_t *ctr) {
  __shared__ uint32_t s_part[kFoldWarps], s_sum[2][kFoldWarps];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t *err = ctr + kFoldErr;
  uint32_t target = 0, count = 1, base = 0, levels = 0;
  int32_t *fr = fr0, *next = fr1;  // fr0[0] is the root pair, 0
  while (count > 0) {
    if ((uint64_t)base + count > cap || levels >= 128) {
      if (blockIdx.x == 0 && tid == 0) atomicOr(err, 4u);
      return;
    }
    const uint32_t run = (count + gridDim.x - 1) / gridDim.x;
    const uint32_t beg = min(count, blockIdx.x * run), end = min(count, beg + run);
    uint32_t mine = 0;
    for (uint32_t f = beg + tid; f < end; f += kFoldThreads) {
      const uint32_t c = expand_node(bvh2, n_pairs, __ldcg(fr + f), bvh8 + 16ull * (base + f), choice, err);
      inner_cnt[f] = c;
      mine += c;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) s_part[warp] = mine;
    __syncthreads();
    if (warp == 0) {
      mine = __reduce_add_sync(0xffffffffu, lane < kFoldWarps ? s_part[lane] : 0u);
      if (lane == 0) counts[blockIdx.x] = mine;
    }
    if (!grid_barrier_bit(ctr + kFoldBarrier, err, kFoldTimeout, target)) return;
    uint32_t before = 0, total = 0;
    for (uint32_t b = tid; b < gridDim.x; b += kFoldThreads) {
      const uint32_t c = __ldcg(counts + b);
      total += c;
      if (b < blockIdx.x) before += c;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    total = __reduce_add_sync(0xffffffffu, total);
    if (lane == 0) s_sum[0][warp] = before, s_sum[1][warp] = total;
    __syncthreads();
    before = __reduce_add_sync(0xffffffffu, lane < kFoldWarps ? s_sum[0][lane] : 0u);
    total = __reduce_add_sync(0xffffffffu, lane < kFoldWarps ? s_sum[1][lane] : 0u);
    const uint32_t next_base = base + count;
    if ((uint64_t)next_base + total > cap) {
      if (blockIdx.x == 0 && tid == 0) atomicOr(err, 4u);
      return;  // every CTA: the same sums
    }
    for (uint32_t f0 = beg; f0 < end; f0 += kFoldThreads) {
      const uint32_t f = f0 + tid;
      const uint32_t c = f < end ? inner_cnt[f] : 0u;  // this thread's own write
      uint32_t x = c;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      __syncthreads();
      if (lane == 31) s_part[warp] = x;
      __syncthreads();
      const uint32_t part = lane < kFoldWarps ? s_part[lane] : 0u;
      uint32_t r = before + x - c + __reduce_add_sync(0xffffffffu, lane < warp ? part : 0u);
      before += __reduce_add_sync(0xffffffffu, part);
      if (c == 0) continue;
      float4 *o = bvh8 + 16ull * (base + f);
      for (int s = 0; s < 8; s++) {
        const int32_t ref = __float_as_int(o[2 * s + 1].z);
        if (ref < 0) continue;
        next[r] = ref;
        o[2 * s + 1].z = __int_as_float((int32_t)(next_base + r));
        r++;
      }
    }
    base = next_base;
    count = total;
    levels++;
    int32_t *t = fr;
    fr = next;
    next = t;
    if (!grid_barrier_bit(ctr + kFoldBarrier, err, kFoldTimeout, target)) return;
  }
  if (blockIdx.x == 0 && tid == 0) {
    ctr[kFoldNodes] = base;
    ctr[kFoldLevels] = levels;
  }
}

// fp32 fold -> 96-byte quantized nodes, every child ref range-checked (inner
// refs against the node count, leaf refs against the triangle count): the
// traversal uses leaf refs without a check.
__global__ void k_quantize8(const float4 *__restrict__ wide, const uint32_t *__restrict__ n8_at, uint32_t ntris,
                            uint4 *__restrict__ out, uint32_t *__restrict__ err) {
  const uint32_t n8 = *n8_at;
  for (uint32_t f = blockIdx.x * blockDim.x + threadIdx.x; f < n8; f += gridDim.x * blockDim.x) {
    const float4 *W = wide + 16ull * f;
    float box[8][6];
    int32_t ref[8];
    uint32_t fmask = 0;
    for (int s = 0; s < 8; s++) {
      const float4 a = W[2 * s], b = W[2 * s + 1];
      box[s][0] = a.x, box[s][1] = a.y, box[s][2] = a.z;
      box[s][3] = a.w, box[s][4] = b.x, box[s][5] = b.y;
      ref[s] = __float_as_int(b.z);
      if (ref[s] == INT_MIN) continue;
      fmask |= 1u << s;
      if (ref[s] < 0 ? (uint32_t)~ref[s] >= ntris : (uint32_t)ref[s] >= n8) atomicOr(err, 2u);
    }
    uint32_t w[24];
    if (!quantize_node8(box, ref, fmask, w)) atomicOr(err, 8u);
    uint4 *o = out + 6ull * f;
    for (int i = 0; i < 6; i++) o[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
}

}  // namespace

uint32_t bvh8_capacity(uint32_t ntris) { return ntris ? (uint32_t)((4ull * ntris + 6) / 7 + 1) : 0; }

namespace {

// The SAH choices of every pair (k_collapse_costs) into `choice`; `scr`
// holds 10 words per pair plus one per leaf.
cudaError_t collapse_choices(const DevScene &d, uint32_t *scr, uint32_t *choice, uint32_t *errw, cudaStream_t st) {
  const uint32_t n_pairs = d.ntris - 1;
  int32_t *parent = (int32_t *)scr, *leaf_parent = (int32_t *)(scr + n_pairs);
  uint32_t *arrivals = scr + n_pairs + d.ntris;
  float *cost = (float *)(arrivals + n_pairs);
  cudaError_t e = cudaMemsetAsync(parent, 0xff, 4ull * (n_pairs + d.ntris), st);  // parent, leaf_parent: -1
  if (e == cudaSuccess) e = cudaMemsetAsync(arrivals, 0, 4ull * n_pairs, st);
  if (e != cudaSuccess) return e;
  k_pair_parents<<<(n_pairs + 255) / 256, 256, 0, st>>>(d.bvh2, n_pairs, parent, leaf_parent, d.ntris, errw);
  k_collapse_costs<<<(d.ntris + 255) / 256, 256, 0, st>>>(d.bvh2, n_pairs, d.ntris, parent, leaf_parent, arrivals,
                                                          cost, choice, errw);
  return cudaGetLastError();
}

}  // namespace

cudaError_t build_bvh8(const DevScene &d, bool sah, void *bvh8q, uint32_t cap, uint32_t *n8_out,
                       uint32_t *levels_out, int32_t *root_out, char *errbuf, size_t errlen, ScratchPool &pool,
                       cudaStream_t st) {
  *n8_out = 0;
  *levels_out = 0;
  *root_out = 0;  // node 0
  if (d.ntris == 0 || cap == 0 || !bvh8q) return cudaErrorInvalidValue;
  const bool leaf_root = d.root_ref < 0;  // one triangle: a single node with the root leaf in slot 0
  const uint32_t n_pairs = leaf_root ? 0 : d.ntris - 1;
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fold8, kFoldThreads, 0);
  if (e != cudaSuccess) return e;
  const uint32_t grid = std::max(1u, std::min((uint32_t)(sms * std::max(1, std::min(per_sm, 4))),
                                              (cap + kFoldThreads - 1) / kFoldThreads));
  // Scratch: the fp32 nodes (256 bytes each), control words, two frontiers and
  // the inner counts (cap words each), the CTAs' counts; for the SAH the
  // pairs' choices, and for their computation the parent links, arrival
  // counters and costs (11 words per pair, 1 per leaf).
  const size_t sah_words = sah && !leaf_root ? 11ull * n_pairs + d.ntris : 0;
  const size_t words = 64ull * cap + 64 + 3ull * cap + grid + sah_words;
  uint32_t *mem = nullptr;
  if ((e = scratch_alloc((void **)&mem, 4 * words, pool, st)) != cudaSuccess) return e;
  float4 *wide = reinterpret_cast<float4 *>(mem);
  uint32_t *ctr = mem + 64ull * cap;
  int32_t *fr0 = reinterpret_cast<int32_t *>(ctr + 64), *fr1 = fr0 + cap;
  uint32_t *cnt = reinterpret_cast<uint32_t *>(fr1 + cap), *counts = cnt + cap;
  uint32_t *choice = sah && !leaf_root ? counts + grid : nullptr;
  uint32_t h[kFoldWords] = {0};
  auto fold = [&](uint32_t *ch) {
    cudaError_t r = cudaMemsetAsync(ctr, 0, 4 * kFoldWords, st);
    if (leaf_root) {
      auto bits = [](int32_t i) {
        float f;
        std::memcpy(&f, &i, 4);
        return f;
      };
      float4 node[16];
      const float inf = bits(0x7f800000);
      for (int s = 0; s < 8; s++) {
        node[2 * s] = make_float4(inf, inf, inf, inf);
        node[2 * s + 1] = make_float4(inf, inf, bits(INT_MIN), 0.0f);
      }
      node[0] = make_float4(d.root_lo[0], d.root_lo[1], d.root_lo[2], d.root_hi[0]);
      node[1] = make_float4(d.root_hi[1], d.root_hi[2], bits(d.root_ref), 0.0f);
      const uint32_t one[2] = {1u, 1u};
      if (r == cudaSuccess) r = cudaMemcpyAsync(wide, node, sizeof(node), cudaMemcpyHostToDevice, st);
      if (r == cudaSuccess) r = cudaMemcpyAsync(ctr + kFoldNodes, one, sizeof(one), cudaMemcpyHostToDevice, st);
    } else {
      if (r == cudaSuccess) r = cudaMemsetAsync(fr0, 0, 4, st);  // the root pair is bvh2 record 0
      if (r == cudaSuccess && ch) r = collapse_choices(d, ch + n_pairs, ch, ctr + kFoldErr, st);
      if (r != cudaSuccess) return r;
      const float4 *bvh2 = d.bvh2;
      uint32_t np = n_pairs, cp = cap;
      const uint32_t *cc = ch;
      void *args[] = {&bvh2, &np, &cc, &wide, &cp, &fr0, &fr1, &cnt, &counts, &ctr};
      r = cudaLaunchCooperativeKernel((const void *)k_fold8, dim3(grid), dim3(kFoldThreads), args, 0, st);
    }
    if (r != cudaSuccess) return r;
    k_quantize8<<<(uint32_t)std::min<uint64_t>(((uint64_t)cap + 127) / 128, (uint64_t)sms * 16), 128, 0, st>>>(
        wide, ctr + kFoldNodes, d.ntris, static_cast<uint4 *>(bvh8q), ctr + kFoldErr);
    r = cudaGetLastError();
    if (r == cudaSuccess) r = cudaMemcpyAsync(h, ctr, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (r == cudaSuccess) r = cudaStreamSynchronize(st);
    return r;
  };
  e = fold(choice);
  // The SAH fold has no node bound below one per pair: past the capacity
  // sized for the largest-first fold, take that fold instead.
  if (e == cudaSuccess && choice && (h[kFoldErr] & 4u)) e = fold(nullptr);
  cudaFreeAsync(mem, st);
  if (e != cudaSuccess) return e;
  const uint32_t bad = h[kFoldErr], n8 = h[kFoldNodes];
  if (bad || n8 >= (1u << 28)) {
    if (bad & 8u)
      snprintf(errbuf, errlen, "bvh8: a child box does not fit its node's 8-bit grid");
    else
      snprintf(errbuf, errlen, "bvh8 collapse: %s",
               bad & kFoldTimeout ? "device wait timed out"
                                  : (bad & 3u ? "bad child reference" : "node capacity exceeded"));
    return cudaErrorInvalidValue;
  }
  *n8_out = n8;
  *levels_out = h[kFoldLevels];
  return cudaSuccess;
}

}  // namespace rtgb

// Host forms of the node quantization and the octant slot assignment, so
// that the containment guarantee and the fold can be checked without a GPU
// (rt_scenes.h).
extern "C" uint32_t rtgbQuantizeNode8(const float *boxes, const int32_t *refs, uint32_t fmask, uint32_t *out) {
  fmask &= 0xffu;
  if (!boxes || !refs || !out || fmask == 0) return 0;
  float box[8][6] = {};
  int32_t ref[8];
  for (uint32_t s = 0; s < 8; s++) {
    const bool f = (fmask >> s) & 1u;
    ref[s] = f ? refs[s] : INT_MIN;
    for (int j = 0; j < 6; j++) box[s][j] = f ? boxes[6 * s + j] : 0.0f;
  }
  return rtgb::quantize_node8(box, ref, fmask, out) ? 1u : 0u;
}

extern "C" uint32_t rtgbAssignOctantSlots(const float *boxes, uint32_t cnt, int32_t *slot_of) {
  if (!boxes || !slot_of || cnt < 1 || cnt > 8) return 0;
  float box[8][6] = {};
  for (uint32_t i = 0; i < cnt; i++)
    for (int j = 0; j < 6; j++) box[i][j] = boxes[6 * i + j];
  int so[8];
  rtgb::assign_octant_slots(box, (int)cnt, so);
  for (uint32_t i = 0; i < cnt; i++) slot_of[i] = so[i];
  return 1;
}
