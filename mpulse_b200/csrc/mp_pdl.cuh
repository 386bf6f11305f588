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

// pdl_launch_dependents lets the next kernel of the stream start its blocks once
// all of this kernel's have called it or ended; pdl_wait waits until the previous
// kernel's writes are visible.  Both are no-ops for a kernel launched without the
// attribute.  The step kernels call the first when a block has done its planes: called
// at their start, the next kernel's blocks took the register file's room beside them
// and waited there (64^3 FP32 6.9 us a step, at the end 5.8; 48^3 Kerr 7.7 and 6.3;
// 32^3 FP64 4.2 and 3.6).  The reverse kernels, whose set-up is longer, call it at
// their start (96^3 FP32 39.8 us a reverse step, at the end 46.5).
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
