// Kernel launches with programmatic dependent launch.
//
// A chain of the library's kernels is launched so that each may be brought up while the last CTAs of
// the one before it finish: its launch latency, its parameter fetch and the constants it reads are then
// off the chain.  Every kernel launched this way calls pdl_wait before it touches anything an earlier
// kernel reads or writes; it returns once the grids before have completed and their writes are visible.
// Kernels of other libraries in between keep the full order on both sides.  One rotation at N = 2^13,
// level 3: 73 -> 50 us; one product at N = 2^16, level 30: 259 -> 225; a bootstrap: 16.2 -> 14.8 ms.  A
// kernel's dependents come up when its CTAs exit: with griddepcontrol.launch_dependents at its
// beginning the same chains took 61 us, 247 us and 15.9 ms, and a batch of 16 operations 2.70 ms
// instead of 2.56.
#pragma once
#include <cuda_runtime.h>

#include "context.hpp"

namespace fides {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename T>
struct AsDeclared {  // the kernel's own parameter types, not deduced from the arguments
  using type = T;
};
template <typename... P>
void launch_pdl(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s,
                const typename AsDeclared<P>::type&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  void* p[] = {const_cast<void*>(static_cast<const void*>(&args))...};
  const cudaError_t kernel_launch = cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), p);
  if (kernel_launch != cudaSuccess) cudaGetLastError();  // reported here, not by the thread's next check as well
  FIDES_CUDA(kernel_launch);
}

}  // namespace fides
