// t, u, v of a hit in fp64: triIntersect (ray-trace-compute.comp:157-173) of the
// chosen triangle, evaluated once and rounded to fp32, which removes the
// cancellation error the fp32 formula shows at grazing angles.
#pragma once
#include "rt_internal.h"
#include "rt_math.cuh"

namespace rtgb {

struct d3 {
  double x, y, z;
};
__device__ __forceinline__ d3 dsub(d3 a, d3 b) { return d3{__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
__device__ __forceinline__ double ddot(d3 a, d3 b) {
  return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
__device__ __forceinline__ d3 dcross(d3 a, d3 b) {
  return d3{__dsub_rn(__dmul_rn(a.y, b.z), __dmul_rn(b.y, a.z)), __dsub_rn(__dmul_rn(a.z, b.x), __dmul_rn(b.z, a.x)),
            __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(b.x, a.y))};
}

// triIntersect in fp64 on the original vertices (fp32 inputs widened).
__device__ __forceinline__ void refine_fp64(const rt_triangle *__restrict__ tris, int tri, f3 o, f3 d, float &t,
                                            float &u, float &v) {
  const float4 *T = reinterpret_cast<const float4 *>(tris + tri);
  float4 a4 = __ldg(T), b4 = __ldg(T + 1), c4 = __ldg(T + 2);
  d3 v0{a4.x, a4.y, a4.z}, v1{b4.x, b4.y, b4.z}, v2{c4.x, c4.y, c4.z};
  d3 ro{o.x, o.y, o.z}, rd{d.x, d.y, d.z};
  d3 a = dsub(v0, v1), b = dsub(v2, v0), p = dsub(v0, ro);
  d3 n = dcross(b, a);
  d3 q = dcross(p, rd);
  double idet = __ddiv_rn(1.0, ddot(rd, n));
  u = __double2float_rn(__dmul_rn(ddot(q, b), idet));
  v = __double2float_rn(__dmul_rn(ddot(q, a), idet));
  t = __double2float_rn(__dmul_rn(ddot(n, p), idet));
}

}  // namespace rtgb
