// pdl.cuh -- programmatic dependent launch of the step's kernels.
//
// A step is a chain of 9 to 23 short kernels.  Launched with the programmatic
// attribute, a kernel's CTAs come up while its predecessor drains, and wait in
// pdl_enter() until the predecessor has completed and its stores are visible;
// what overlaps is the launch latency alone.  Every kernel of a chain calls
// pdl_enter() in every thread before anything else, also where a case is idle:
// a kernel that completes has then waited for its predecessor, so that waiting
// for the direct predecessor is waiting for all of them.
#pragma once
#include <cuda_runtime.h>

namespace rbc {
namespace dev {

__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace dev

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace rbc
