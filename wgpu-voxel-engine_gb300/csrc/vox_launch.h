// vox_launch.h — launches that overlap their start with the end of the launch before them
// (programmatic dependent launch). The dependent kernel may begin as soon as every CTA of the
// one before it in the stream has called pdl_trigger (or ended), and calls pdl_wait before it
// touches anything that earlier work of the stream writes or reads: the wait ends when all of
// that work is complete and visible. What is saved is the launch latency between dependent
// kernels, about a microsecond each; a kernel that follows one without a trigger starts as usual.
// A kernel whose dependent reads anything before its own pdl_wait triggers after pdl_wait itself
// (or is launched without this attribute), so that everything ahead of both has ended by then.
// What earlier launches write is read behind the wait by plain (or volatile, or acquiring) loads:
// pdl_wait keeps those behind it. No __ldg and no `const __restrict__` pointer for such data: both
// say that it does not change while the kernel runs, which is untrue of a kernel that starts
// early, and let the compiler move the load ahead of the wait. (The other cached-load intrinsics
// give the compiler no order either; they are used where the address depends on an acquired
// value.) Data of the context that no launch writes, such as grad2, may be read by __ldg.
#pragma once

#include <cstring>
#include <cuda_runtime.h>

namespace vox {

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

inline cudaError_t launch_dependent(const void* fn, dim3 grid, dim3 block, void** params, size_t smem,
                                    cudaStream_t stream) {
  cudaLaunchAttribute attr;
  std::memset(&attr, 0, sizeof attr);
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, params);
}

}  // namespace vox
