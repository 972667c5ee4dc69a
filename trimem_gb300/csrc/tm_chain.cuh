// Chains of kernels with programmatic dependent launches: a kernel of a chain
// may start while the one before drains, and waits for its results only
// where it needs them.  What an earlier kernel of the chain writes is read by
// plain loads: read-only loads (const __restrict__, __ldg) may be moved above
// the wait.
#pragma once

#include "tm_internal.h"

namespace tmg {

// waits until the previous kernel of the chain has finished and its writes
// are visible; every kernel of a chain calls it before it touches what an
// earlier one writes, so that completion carries along the chain
__device__ __forceinline__ void wait_previous() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void let_next_start() { cudaTriggerProgrammaticLaunchCompletion(); }

// launch with programmatic stream serialisation (see wait_previous)
template <class... A, class... B>
void launch_after_smem(void (*k)(A...), int grid, int block, size_t smem, cudaStream_t s, B... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TM_CUDA(cudaLaunchKernelEx(&cfg, k, args...));
}
template <class... A, class... B>
void launch_after(void (*k)(A...), int grid, int block, cudaStream_t s, B... args) {
  launch_after_smem(k, grid, block, 0, s, args...);
}

}  // namespace tmg
