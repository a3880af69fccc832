// Kernel launches that may begin while the kernel before them on the stream
// still runs (programmatic dependent launch).
#pragma once

#include <cuda_runtime.h>

namespace atm {

// First statement of every kernel started by launch(): waits until the kernels
// before it on the stream have completed and their writes are visible, then lets
// the next one be set up.  Nothing is read or written before it.
__device__ __forceinline__ void stream_order() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
inline cudaError_t launch(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, A... a) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(a)...);
}

}  // namespace atm
