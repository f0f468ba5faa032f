// Launches of a step's kernels that overlap the launch itself: the next
// kernel's blocks are set up while the last blocks of the previous one run
// (programmatic dependent launch) and wait there for its completion.  A small
// world's step is a chain of kernels of 5 to 25 us, whose launch gaps this
// shortens.
#pragma once

#include <cuda_runtime.h>

namespace phy {

// First statement of a kernel launched with launch_after: everything before
// it in the stream has completed and is visible; then lets the next kernel's
// blocks be set up.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Lets the next kernel's blocks be set up (they still wait for this one).
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Particles below which a step's passes overlap: 1,287 to 36,864 particles gain
// 3 to 6 us a step; at 76,800 (f64) and 379,603 (compensated) the early blocks
// cost 12 and 25 us.
constexpr int kOverlapBelow = 40000;

// `overlap`: whether to; a launch without it starts after the previous kernel.
template <class... P, class... A>
inline void launch_after(bool overlap, void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t s,
                         const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace phy
