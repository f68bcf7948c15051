// wt_launch.cuh -- launches that overlap the end of the kernel before them.
//
// A step is a chain of launches, each reading what the one before wrote.  With
// programmatic stream serialization a kernel's CTAs may be scheduled as soon as
// every CTA of the one before has passed dep_wait() or left: what a kernel does
// before its own dep_wait() -- set-up, mesh tables and metric terms, which only
// synchronous mesh calls write -- then runs under the tail of its predecessor.
// dep_wait() returns when every earlier launch of the chain is complete and its
// writes are visible, so everything a step writes is read or written after it.
// Every thread of such a kernel calls it, early-leaving ones too: a launch is
// then complete only after its predecessor.  After an ordinary launch, and in a
// kernel launched the ordinary way, it does not wait.
//
// Measured (B200): ten SIPG steps on 4^3 elements, n = 6, 357 -> 309 us; one
// right-hand side at n = 7 with dissipation 129 -> 117 us; two Tsit5 steps 24^3 x
// 6^3 3.56 -> 3.42 ms.  Not for the persistent n = 8 kernels: the next launch's
// CTAs then take an SM's room as it frees, unevenly (40^3 FP32 step 6.5 -> 9.0 ms).
#pragma once
#include <cuda_runtime.h>

namespace wt {

__device__ __forceinline__ void dep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The launches of a batch, parallel branches of one graph, gain nothing from it (an
// FP32 batch of 24 small solves 748 us a call so, 703 us with ordinary launches): DEP
// = false launches the ordinary way.
template <bool DEP = true, typename... P, typename... A>
int launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... a) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = DEP ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(a)...) == cudaSuccess ? 0 : -2;
}

// Let a kernel have `bytes` of dynamic shared memory, and (carveout) the SM give shared
// memory all it can, where the kernel's CTAs need it to be resident as planned.  Called
// before each launch: the attributes belong to the current device, and a process may
// have contexts on several, or reset one (under 1 us a call; steps replay a graph).
template <typename K>
int allow_smem(K kernel, size_t bytes, bool carveout = false) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return -2;
  if (carveout && cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess)
    return -2;
  return 0;
}

}  // namespace wt
