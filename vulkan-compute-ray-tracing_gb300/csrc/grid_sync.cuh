// Barrier over a cooperative grid (all CTAs resident: cudaLaunchCooperativeKernel).
#pragma once
#include "rt_internal.h"

namespace rtgb {

// `counter` is zero at launch and only grows; `target` is each thread's own
// count of expected arrivals, zero at launch. A CTA that has polled for far
// longer than any phase takes records an error and gets false, and so do the
// others, at the same or their next barrier: every caller returns on false.
// Data written before the barrier by other CTAs is read past L1 (__ldcg).
__device__ __forceinline__ bool grid_barrier_bit(uint32_t *counter, uint32_t *err, uint32_t bit, uint32_t &target) {
  __shared__ int s_ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1u);
    int ok = 0;
    for (uint32_t poll = 0; poll < (1u << 28); poll++) {
      const uint32_t at = *reinterpret_cast<volatile uint32_t *>(counter);
      if ((int32_t)(at - target) >= 0) {
        ok = 1;
        break;
      }
      if (poll > 64) __nanosleep(32);
    }
    if (!ok) atomicOr(err, bit);
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}
__device__ __forceinline__ bool grid_barrier(uint32_t *counter, uint32_t *err, uint32_t &target) {
  return grid_barrier_bit(counter, err, KERR_TIMEOUT, target);
}

}  // namespace rtgb
