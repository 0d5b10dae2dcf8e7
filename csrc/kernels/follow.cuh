// Launches that are set up while the kernel before them in the stream ends (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace nangila {

// In a kernel launched with launch_following: waits until the kernel before it is complete and its writes are visible. Every thread calls
// it before it touches memory.
__device__ __forceinline__ void follow() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// In the kernel before it: lets the next one be set up from here on (without it, when this CTA ends). Its CTAs then wait on the SMs, so
// not before a wait for another rank.
__device__ __forceinline__ void may_follow() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Args>
cudaError_t launch_following(void (*kernel)(Args...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace nangila
