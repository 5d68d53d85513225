// Traversal of the 8-wide nodes by a whole warp from shared pools, for
// launches whose time is the chain of steps of their longest ray.
//
// A warp holds R rays (2 to 8). The nodes still to visit, of all of them, are
// one pool in shared memory: a step takes the newest 32 entries, one a lane,
// tests each node against its ray (wide.cuh) and puts the entered children
// back, nearer octant ranks on top; hit leaves go to a leaf pool that the
// lanes test 32 at a time. So one ray's pending nodes are visited side by
// side: it takes several times fewer steps than its visits, for more visits
// (nodes that a nearer hit would have pruned). A launch that fills the GPU is
// better off with a ray per lane (k_trace_wide).
//
// The hit is k_trace_wide's: each ray's key (ordered t, triangle) is lowered
// by a shared-memory atomicMin, whatever the order. A ray is done when its
// count of entries in both pools is zero.
#pragma once
#include "rt_internal.h"
#include "wide.cuh"

namespace rtgb {

constexpr int kPoolBlock = 128;
constexpr uint32_t kNodePool = 1024, kLeafPool = 512;
// Below this many pool nodes the lanes would idle: what leaves there are get tested first.
constexpr uint32_t kLeafFlush = 8;
// Pool entries kept free for walking one entry at a time (at most seven
// siblings a level stay behind, over at most 64 levels) and for a root per
// ray: rays start only while the pool is below kNodeRoom.
constexpr uint32_t kNodeRoom = kNodePool - 7 * 64 - 32;

// One warp's rays and pools.
template <int R>
struct PoolWarp {
  float4 org[R], dir[R], inv[R];  // origin and octant; direction and tmin; 1 / direction and tmax
  float4 hit[R];                  // t, u, v, leaf of the key's triangle
  unsigned long long key[R];      // closest hit so far: ordered t, triangle
  uint32_t left[R];               // the ray's entries in both pools
  uint32_t nodes[kNodePool], leaves[kLeafPool];
  uint32_t node_count, leaf_tail, pad[2];
};

__device__ __forceinline__ unsigned long long pool_miss_key(float tmax) {
  return (unsigned long long)ord_f(__fadd_rn(tmax, 0.0f)) << 32;
}

// The ray of slot `slot`: its root goes to the node pool if the ray enters it.
template <int R>
__device__ __forceinline__ void pool_start(PoolWarp<R> &S, const DevScene &sc, uint32_t slot, f3 o, f3 d, float tmin,
                                           float tmax) {
  const TraceRay r = make_ray(o, d, tmin);
  S.org[slot] = make_float4(o.x, o.y, o.z, __int_as_float(ray_octant(r)));
  S.dir[slot] = make_float4(d.x, d.y, d.z, tmin);
  S.inv[slot] = make_float4(r.ix(), r.iy(), r.iz(), tmax);
  S.key[slot] = pool_miss_key(tmax);
  const float root = slab_enter(r, sc.root_lo[0], sc.root_hi[0], sc.root_lo[1], sc.root_hi[1], sc.root_lo[2],
                                sc.root_hi[2], tmax);
  const bool in = root < __int_as_float(0x7f800000);
  S.left[slot] = in ? 1u : 0u;
  if (in) S.nodes[atomicAdd(&S.node_count, 1u)] = ((uint32_t)sc.root8 << 5) | slot;
}

// One step of the warp: up to 32 nodes, then the leaf rounds that are due.
// Every node is numbered above its parent (bvh8.cu), so the steps end.
template <int R>
__device__ __forceinline__ void pool_step(PoolWarp<R> &S, const DevScene &sc, uint32_t lane, uint32_t &head,
                                          uint32_t *err) {
  volatile PoolWarp<R> &V = S;
  uint32_t count = V.node_count;
  const uint32_t take = min(count, min(32u, max(1u, count < kNodeRoom ? (kNodeRoom - count) / 8 : 0u)));
  const uint32_t e = lane < take ? S.nodes[count - 1 - lane] : 0u;
  __syncwarp();
  if (lane == 0) S.node_count = count - take;
  __syncwarp();
  if (lane < take) {
    const uint32_t q = e & 31u, node = e >> 5;
    if (node >= sc.n8) {
      atomicOr(err, KERR_BAD_INDEX);
      atomicSub(&S.left[q], 1u);
    } else {
      const float4 o4 = S.org[q], i4 = S.inv[q];
      TraceRay r;
      r.o = mk3(o4.x, o4.y, o4.z);
      r.ixy = pk2(i4.x, i4.y);
      r.izz = pk2(i4.z, i4.z);
      r.tmin = S.dir[q].w;
      const uint32_t oct = __float_as_uint(o4.w);
      WideStep ws;
      wide_node_test(sc.bvh8, (int)node, r, oct, ord_inv((uint32_t)(V.key[q] >> 32)), ws);
      const uint32_t ci = __popc(ws.hin), cl = __popc(ws.leafmask);
      atomicAdd(&S.left[q], ci + cl - 1u);
      if (ci) {
        const uint32_t at = atomicAdd(&S.node_count, ci), ranks = rank_bits(ws.hin, oct);
#pragma unroll
        for (uint32_t s = 0; s < 8; s++)
          if ((ws.hin >> s) & 1u) S.nodes[at + __popc(ranks >> ((s ^ oct) + 1u))] = ((uint32_t)ws.ref[s] << 5) | q;
      }
      if (cl) {
        uint32_t at = atomicAdd(&S.leaf_tail, cl);
#pragma unroll
        for (uint32_t s = 0; s < 8; s++)
          if ((ws.leafmask >> s) & 1u) S.leaves[at++ & (kLeafPool - 1)] = ((uint32_t)~ws.ref[s] << 5) | q;
      }
    }
  }
  __syncwarp();
  count = V.node_count;
  const uint32_t tail = V.leaf_tail;
  while (tail - head >= 32u || (tail != head && count < kLeafFlush)) {
    const uint32_t cnt = min(tail - head, 32u);
    bool acc = false;
    unsigned long long cand = 0;
    uint32_t owner = 0;
    int k = 0;
    float ct = 0.0f, cu = 0.0f, cv = 0.0f;
    if (lane < cnt) {
      const uint32_t l = S.leaves[(head + lane) & (kLeafPool - 1)];
      owner = l & 31u;
      k = (int)(l >> 5);
      const uint32_t tri = (uint32_t)__ldg(sc.leaf_tri + k);
      const float4 q0 = S.org[owner], q1 = S.dir[owner];
      const unsigned long long cur = V.key[owner];
      if (tri_candidate(sc.tpre, k, mk3(q0.x, q0.y, q0.z), mk3(q1.x, q1.y, q1.z), q1.w,
                        ord_inv((uint32_t)(cur >> 32)), ct, cu, cv)) {
        const unsigned long long key =
            ((unsigned long long)ord_f(__fadd_rn(ct, 0.0f)) << 32) | tri;
        if (key < cur) {
          acc = true;
          cand = key;
          atomicMin(&S.key[owner], key);
        }
      }
      atomicSub(&S.left[owner], 1u);
    }
    __syncwarp();
    if (acc && V.key[owner] == cand) S.hit[owner] = make_float4(ct, cu, cv, __int_as_float(k));
    __syncwarp();
    head += cnt;
  }
}

}  // namespace rtgb
