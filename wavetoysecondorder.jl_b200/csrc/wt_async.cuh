// wt_async.cuh -- per-thread asynchronous copies global -> shared (cp.async).
#pragma once
#include "wt_common.cuh"

namespace wt {

// Per-thread asynchronous copy of one word (4 or 8 bytes) global -> shared,
// and the wait for all of this thread's copies.  The generic kernels copy the
// words their node pass reads at their own node (coefficients, Pi, RK state)
// at kernel start, so that those loads run under the contraction; each thread
// reads back only its own words, so the wait needs no CTA barrier.
template <typename T>
__device__ __forceinline__ void cp_async_word(T* dst, const T* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_own() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// ends a group of copies; wait until at most `n` of the thread's newest groups are in flight
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int n>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(n) : "memory"); }

}  // namespace wt
