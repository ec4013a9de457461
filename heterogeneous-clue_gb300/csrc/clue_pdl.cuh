// Programmatic dependent launch: the kernels of one run are queued so that
// each lets the next one's blocks onto the device as soon as all its own have
// started (pdl_trigger) and waits for the whole previous kernel before it
// touches memory (pdl_wait), so that a stage starts without a launch's
// latency.  A kernel's completion implies its predecessors', since each waits
// before it ends.  The first kernel of a run is launched the ordinary way, and
// the last one triggers nothing: work before and after a run on the stream
// sees ordinary kernels.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace clue {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_trigger();
}

// Queues a kernel that begins with pdl_wait().
template <class... Params, class... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                       Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace clue
