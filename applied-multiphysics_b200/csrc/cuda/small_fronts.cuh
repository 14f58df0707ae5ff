// Shared by the whole-front kernels (front_small.cu for FP64 factors, front_small_f32.cu for FP32 ones).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "../host/plan.hpp"

namespace amp {

// Tiny fronts come in two size classes (sorted by m within each level by the plan): m <= kTinyMid with 8 warps per
// CTA and 16 x 16 tiles, and kTinyMid < m <= 32 with 4 warps per CTA and 32 x 32 tiles, so that the many smallest fronts
// are not held to the shared memory of the largest.
template <int MAXM>
constexpr int tiny_warps() {
  return MAXM <= kTinyMid ? 8 : 4;
}

template <int G>
__device__ __forceinline__ void group_sync() {
  if constexpr (G == 32)
    __syncwarp();
  else
    __syncthreads();
}

// |d| < tau (or NaN) becomes -tau / +tau by the sign of d; a non-finite small pivot fails (ldlt.mjs:513-522)
template <class TC>
__device__ __forceinline__ bool small_ldlt_pivot(TC &d, TC tau, int &neg, int &pert) {
  if (!(fabs(d) >= tau)) {
    if (!isfinite(d)) return false;
    d = d < TC(0) ? -tau : tau;
    pert++;
  }
  if (d < TC(0)) neg++;
  return true;
}

// Children of one front whose metadata a CTA holds at a time (fetched in parallel, applied in the reference's order)
constexpr int kChildChunk = 32;
struct ChildMeta {
  int muc[kChildChunk];
  int64_t uo[kChildChunk], ea[kChildChunk];
};

}  // namespace amp
