// launch.h -- launches with programmatic serialisation: the kernel's CTAs may
// start before the kernel ahead of it in the stream has ended.  For kernels
// that wait for it themselves (grid_dependency_wait, chain_begin) before they
// touch memory that it, or one ahead of it, reads or writes.
#pragma once

#include <cuda_runtime.h>

namespace medimg {

template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                             Args &&...args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace medimg
