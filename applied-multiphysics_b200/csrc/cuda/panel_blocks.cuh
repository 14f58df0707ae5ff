// Shared by the group panels (group_panel.cu, cgroup_panel.cu): 64 x 64 blocks in shared memory, the warps' row groups, the
// flags between the strips of a launch.
#pragma once
#include <cuda_runtime.h>

#include "../host/plan.hpp"
#include "devplan.cuh"
#include "sync.cuh"

namespace amp {

__device__ __forceinline__ bool panel_failed(const unsigned long long *st) {
  return *(volatile const unsigned long long *)st != kStatusOk;
}

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

// Wait (thread 0, bounded) until *p >= need; false when the factorization has failed (a pivot, or a wait that ran
// out: status set). Thread 0 decides and the CTA follows it after the barrier, so every thread returns the same.
__device__ __forceinline__ bool panel_wait(const int *p, int need, unsigned long long *status, long long limit) {
  __shared__ int ok;
  if (threadIdx.x == 0) {
    long long spins = 0;
    int v = 1;
    while (ld_acquire(p) < need) {
      if (panel_failed(status)) {
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
    if (panel_failed(status)) v = 0;  // a failed pivot also releases its flag
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
