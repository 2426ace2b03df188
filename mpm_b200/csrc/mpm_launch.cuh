// mpm_launch.cuh -- launches of a step's dependent kernels.
//
// Each kernel of a step needs all of the one before it.  A plain launch starts
// a kernel's blocks only after the previous grid has drained and its writes
// are flushed, 2 to 3 us apart on a B200 even inside a CUDA graph; a run of a
// few thousand particles spends most of its time there.  With programmatic
// dependent launch the blocks are scheduled while the previous grid's last
// blocks run and wait on the device (after_previous) for its completion and
// flush.
#pragma once

#include <cuda_runtime.h>

namespace mpm_b200 {

// First statement of every kernel launched with launch_dependent, before any
// access to global memory: lets the next grid of the stream be scheduled and
// waits until the previous one has completed and its writes are visible.  Every
// thread calls it, so a grid that has completed implies all before it have.
// Without effect on a plain launch's order, but not free in a block
// that has little else to do (p2g_dependent).
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// (dependent false: a plain launch)
template <class... P, class... A>
inline void launch_kernel(bool dependent, void (*kernel)(P...), unsigned grid, unsigned block,
                          size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = dependent ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);  // an error stays for the caller's cudaGetLastError
}
template <class... P, class... A>
inline void launch_dependent(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                             cudaStream_t st, const A&... args) {
  launch_kernel(true, kernel, grid, block, smem, st, args...);
}

}  // namespace mpm_b200
