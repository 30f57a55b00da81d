// Programmatic dependent launches: a kernel of a chain is placed while the one
// before it drains, instead of after it. Every kernel that may be launched this
// way calls dependent_launch_wait() before it touches anything the chain
// writes, in every thread that does so and in at least one thread whatever the
// input, so completion passes down the chain. In an ordinary launch both
// instructions do nothing.
#pragma once

#include <cuda_runtime.h>

#include "jc_common.h"

namespace jc {
namespace dev {

__device__ __forceinline__ void dependent_launch_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace dev

// k as a programmatic dependent of the launch before it on `s` (a kernel), or
// as an ordinary launch.
template <typename... P, typename... A>
inline void launch_chained(bool dependent, cudaStream_t s, dim3 blocks, uint32_t threads, size_t smem,
                           void (*k)(P...), A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = blocks;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = dependent ? 1 : 0;
  JC_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k, (P)args...));
}

}  // namespace jc
