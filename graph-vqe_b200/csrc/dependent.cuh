// Kernels that start while the one before them in the stream ends.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace vqemps {

// Dependent launches (programmatic stream serialization): a kernel launched by launch_dependent may start
// while the one before it in the stream still runs, once all of that one's CTAs have called dependents_launch
// or ended. What it reads of earlier kernels' results, and what they may still read, it touches after
// dependency_wait only (a no-op under a plain launch). Every kernel of a chain waits, so a wait covers the whole
// chain; the first one of a call is launched plainly.
// Most kernels do without dependents_launch: it lets the next kernel's CTAs start early, but all on the few SMs that
// have room just then (a training step 728 us plain, 896 with it, 685 without; a gradient of 40 qubits 309 with it,
// 281 without). A partition set's levels, whose CTAs first stage a site each, gain by it (766 us without, 627 with).
__device__ __forceinline__ void dependents_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace vqemps
