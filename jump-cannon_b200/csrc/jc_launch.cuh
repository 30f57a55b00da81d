// Programmatic dependent launches: a kernel of a chain is placed while the one
// before it drains, instead of after it. Every kernel that may be launched this
// way calls dependent_launch_wait() before it touches anything the chain
// writes, in every thread that does so and in at least one thread whatever the
// input, so completion passes down the chain. In an ordinary launch both
// instructions do nothing.
//
// A dependent lives while the kernels before it still store, so for it their
// output is not read-only data: it is read by ordinary loads (never __ldg or
// ld.global.nc) and through pointers without __restrict__, which would allow
// the compiler both, and a load moved above the wait. Only what the chain does not
// write before the kernel (graphs, degrees, the positions until the last kernel
// moves them) goes through the read-only path.
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
// as an ordinary launch. carveout: the shared memory to set aside on an SM, in
// percent, or -1 for the driver's choice.
template <typename... P, typename... A>
inline void launch_chained(bool dependent, int carveout, cudaStream_t s, dim3 blocks, uint32_t threads, size_t smem,
                           void (*k)(P...), A... args) {
  cudaLaunchAttribute at[2]{};
  unsigned n = 0;
  if (dependent) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (carveout >= 0) {
    at[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[n++].val.sharedMemCarveout = (unsigned)carveout;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = blocks;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = n;
  JC_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k, (P)args...));
}

template <typename... P, typename... A>
inline void launch_chained(bool dependent, cudaStream_t s, dim3 blocks, uint32_t threads, size_t smem, void (*k)(P...),
                           A... args) {
  launch_chained(dependent, -1, s, blocks, threads, smem, k, args...);
}

}  // namespace jc
