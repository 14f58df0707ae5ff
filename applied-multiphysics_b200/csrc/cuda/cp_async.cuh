// Asynchronous copies of single elements into shared memory, in groups.
#pragma once
#include <cuda_runtime.h>

namespace amp {

// 4, 8 or 16 bytes (both addresses aligned to them); zeros where the source is not valid (it is not read then)
template <int BYTES>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, bool valid = true) {
  static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async sizes");
  const unsigned to = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? BYTES : 0;
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(gmem), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(to), "l"(gmem), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>  // all but the newest N groups of this thread have arrived
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

}  // namespace amp
