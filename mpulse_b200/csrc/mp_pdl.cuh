// mp_pdl.cuh - programmatic dependent launch, used by the kernels that follow
// one another on a stream step after step.
//
// A kernel launched with launch_pdl may start its blocks before the previous
// kernel of the stream has finished; it does its set-up and waits
// (pdl_wait) before it reads anything an earlier kernel wrote or writes
// anything.  Every kernel of such a chain waits, so the end of one is the end of
// all before it.
#ifndef MPB_MP_PDL_CUH
#define MPB_MP_PDL_CUH

#include <cuda_runtime.h>

namespace mpb {

// Let the next kernel of the stream start its blocks once all of this kernel's
// have started, and wait until the previous kernel's writes are visible.  Both
// are no-ops for a kernel launched without the attribute.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 g, dim3 b, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = g;
  cfg.blockDim = b;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace mpb

#endif
