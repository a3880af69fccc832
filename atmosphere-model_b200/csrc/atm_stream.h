// Kernel launches that may begin while the kernel before them on the stream
// still runs (programmatic dependent launch).
#pragma once

#include <cuda_runtime.h>

namespace atm {

// First statement of every kernel started by launch(): waits until the kernels
// before it on the stream have completed and their writes are visible, then lets
// the next one be set up.  Nothing is read or written before it: the kernel's
// parameters carry no __restrict__, and nothing after it is read by __ldg or
// ld.global.nc but constant tables, as a compiler may take such a load for one of
// memory that never changes and move it above the wait.  What gains from the promise
// that its pointers do not overlap is a function of its own, called after the wait
// (interior_rows, remap_energy_adj_block).
__device__ __forceinline__ void stream_order() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches of up to four times the threads the GPU holds overlap the end of the
// kernel before them; larger ones, whose set-up is nothing beside their work, do
// not.  Measured on B200 (ms a pass: none early / up to 2, 4, 8 times the
// threads): 64x64x20 0.68 / 0.58 0.58 0.58, 251x187x27 1.75 / 1.67 1.65 1.65,
// mixed 150x130x48 1.43 / 1.32 1.30 1.30, two steps of FP64 at 1024x1024x64 32.73 /
// 32.59 32.57 33.01 and of the mixed form 25.41 / 25.12 25.14 25.90.
constexpr unsigned long long EARLY_THREADS = 4ULL * 148 * 2048;

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
  cfg.numAttrs = (unsigned long long)grid.x * grid.y * grid.z * threads <= EARLY_THREADS ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(a)...);
}

}  // namespace atm
