// launch.cuh -- launches of kernels that follow one another on a stream.
//
// A step of a small box takes about as long as the gap between two launches
// (10x10x50 FP64: 4.1 us from step to step of a replayed graph, of which about
// 2.3 us are the kernel).  Kernels launched with `chained` may be set up while
// the kernel before them still runs (programmatic dependent launch): their
// blocks come up on the SMs, wait in chain_begin() until everything the kernel
// before them wrote is there, and let the next kernel come up in turn.  What
// does not begin with chain_begin() is launched the ordinary way.
//
// A chained kernel starts before its inputs are written, so it must not read
// them through the read-only cache: ld_pop (checked.cuh) is a plain load that
// stays behind chain_begin().
#pragma once
#include <cuda_runtime.h>

namespace lbx {

#ifdef __CUDACC__
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

}  // namespace lbx
