// Launch with programmatic dependence on the kernel before it in the stream: the next kernel's CTAs may start (barriers,
// tensor memory, tables) while the one before still runs, and wait in wait_for_previous (tensor_common.cuh) before they
// touch global memory.  A call of small batches is a chain of such launches: step of 16 x 12 tokens 83.0 -> 78.6 us, policy
// step of 16 environments 227 -> 199, of 8192 1170 -> 1130, a sequence of 5 x 67 x 11 188 -> 164.
// Not for the float32 step (split_kernels.cu), whose kernels read before they wait; it launches its own chain.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "bnb_trunk.h"
#include "launch_count.h"

namespace bnb {
template <class... P, class... A>
inline int launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  if (cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...) == cudaSuccess) return BNB_OK;
  (void)cudaGetLastError();
  return BNB_ERR_LAUNCH;
}
}  // namespace bnb
