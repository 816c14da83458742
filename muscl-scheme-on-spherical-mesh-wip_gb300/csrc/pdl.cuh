// Programmatic dependent launch, shared by the step's kernels.
//
// The step's kernels are launched with programmatic stream serialization: a
// kernel may start while its predecessor drains, loads what does not depend
// on it (stencil indices, geometry), then waits in griddep_wait() for the
// predecessor grid to complete and its writes to be visible.  Every read of
// state and every write comes after the wait, so no kernel overwrites what
// its predecessor is still reading.  Without a programmatic predecessor the
// wait returns at once.  launch_dependents lets the next kernel start as soon
// as every block of this one has begun.
#pragma once

#include <cuda_runtime.h>

namespace splash {

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }

// A launch with programmatic stream serialization.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// The first error of a sequence of launches.
struct FirstError {
  cudaError_t e = cudaSuccess;
  void operator()(cudaError_t r) {
    if (e == cudaSuccess) e = r;
  }
  cudaError_t status() const { return e != cudaSuccess ? e : cudaGetLastError(); }
};

}  // namespace splash
