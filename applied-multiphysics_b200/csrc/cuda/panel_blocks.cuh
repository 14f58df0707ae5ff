// Shared by the group panels (group_panel.cu, cgroup_panel.cu): 64 x 64 blocks in shared memory, the warps' row groups, the
// flags between the strips of a launch.
#pragma once
#include <cuda_runtime.h>

#include "../host/plan.hpp"
#include "devplan.cuh"
#include "sync.cuh"

namespace amp {

// 64 x 64 FP64 blocks in shared memory, row-major, the column pairs of row r permuted by a bijection of r mod 8 so that
// the 16-byte accesses of a fragment (8 rows, 4 neighbouring pairs) and the 8-byte stores of the block loads (8 rows,
// 4 columns) touch every bank equally often.
__device__ __forceinline__ int sw(int r, int c) {
  return r * kPanel + (((c >> 1) ^ (((r & 1) << 2) | ((r >> 1) & 3))) << 1) + (c & 1);
}
__device__ __forceinline__ double2 pair_at(const double *S, int r, int c) {  // entries (r, c), (r, c + 1), c even
  return *reinterpret_cast<const double2 *>(S + sw(r, c));
}
__device__ __forceinline__ void set_pair(double *S, int r, int c, double x, double y) {
  *reinterpret_cast<double2 *>(S + sw(r, c)) = make_double2(x, y);
}

// the 8-row group of a warp: the pairs of warps that share a scheduler (w, w + 4) get groups that sum to 7, so the
// lower triangle's work is the same on all four
__device__ __forceinline__ int row_group(int warp) { return warp < 4 ? warp : 11 - warp; }

// What a pivot block's Linv holds: the inverses of the 8 x 8 diagonal blocks of L (64 entries each, one plane or two), and a
// bit per block, those of the first four and of the last four in one int each: set where the rows below are to be solved by
// substitution. The product of a row c with the computed inverse X leaves a residual of some eps |L||X||L| |w| in place of
// substitution's eps |L| |w| (w the solved row), so its error is that of substitution only where |L||X| is small. The bound
// on it is G = max |X(i, j)| r(j), X and the row norms r those of the block scaled as a Cholesky factor (L sqrt|D|): 1 for
// the identity, whatever the rows' and columns' scales, about the square root of the condition of the pivots' matrix with a
// unit diagonal. Blocks with G above kInvBound are substituted. Dense LDL^T fronts of 330 columns whose 8 x 8 blocks reach
// G = 1, 5, 52, 2,700 and 190,000 had errors of 0.03, 0.03, 0.04, 0.7 and 41 with products alone (in units of 336 eps
// |L||D||L|^T; complex ones reached 1,100), at most 0.04 by substitution. Elasticity and heat systems stay below 4; of the
// blocks of the edge-element systems with 10 to 16 elements per edge (LDL^T without interchanges) 1 to 6% are above 16, up
// to 200. The bound and the choice cost the cases 0.2 to 0.7%.
constexpr double kInvBound = 16.0;
// this warp's part of the bits: a lane per column of the blocks, eight lanes to a block
__device__ __forceinline__ void put_wild(double *Linv, int planes, bool wild) {
  const unsigned b = __ballot_sync(0xffffffffu, wild);
  int bits = 0;
#pragma unroll
  for (int p = 0; p < 4; p++) bits |= (b >> (8 * p) & 0xffu) != 0 ? 1 << p : 0;
  if ((threadIdx.x & 31) == 0) reinterpret_cast<int *>(Linv + 512 * planes)[threadIdx.x >> 5] = bits;
}
__device__ __forceinline__ int wild_blocks(const double *Linv, int planes) {
  const int2 v = __ldcg(reinterpret_cast<const int2 *>(Linv + 512 * planes));
  return v.x | v.y << 4;
}

// Wait (thread 0, bounded) until *p >= need; false when the factorization has failed (a pivot, or a wait that ran
// out: status set). Thread 0 decides and the CTA follows it after the barrier, so every thread returns the same.
__device__ __forceinline__ bool panel_wait(const int *p, int need, unsigned long long *status, long long limit) {
  __shared__ int ok;
  if (threadIdx.x == 0) {
    long long spins = 0;
    int v = 1;
    while (ld_acquire(p) < need) {
      if (factor_failed(status)) {
        v = 0;
        break;
      }
      if (++spins > limit) {
        atomicMin(status, status_word(0x7fffffff, 3, 0));
        v = 0;
        break;
      }
      __nanosleep(32);
    }
    if (factor_failed(status)) v = 0;  // a failed pivot also releases its flag
    ok = v;
  }
  __syncthreads();
  return ok != 0;
}

// Publish *p = v after this CTA's global writes: all threads pass the barrier first, and thread 0's release store
// orders every write made before the barrier (by any thread of the CTA) before the flag, for a reader that acquires it.
__device__ __forceinline__ void panel_release(int *p, int v) {
  __syncthreads();
  if (threadIdx.x == 0) st_release(p, v);
}

}  // namespace amp
