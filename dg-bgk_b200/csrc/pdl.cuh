// Programmatic dependent launch, shared by the steps and the network.
#pragma once
#include <cuda_runtime.h>

namespace dgbgk {

// The next kernel of the stream may start (its CTAs as this one's leave their
// SMs) once every CTA has called this or left; what it then does before
// grid_wait must not touch anything an earlier kernel writes.
__device__ __forceinline__ void grid_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// ... and waits here until the kernels before it are complete
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with programmatic dependence on the kernel before it in the stream
// (the kernel waits by itself, grid_wait): its launch and everything it does
// before that wait pass while the other one ends.  The caller looks at
// cudaGetLastError.
template <class... P, class... A>
void launch_pdl(void (*fn)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, fn, args...);
}

}  // namespace dgbgk
