// alloc_retry.h -- an allocation that fails for want of memory is made once more
// after what the library keeps has been given back.
#pragma once

#include <cuda_runtime_api.h>

namespace medimg {

template <typename Alloc, typename GiveBack>
cudaError_t alloc_or_give_back(Alloc &&alloc, GiveBack &&give_back) {
  const cudaError_t e = alloc();
  if (e != cudaErrorMemoryAllocation) return e;
  give_back();
  return alloc();
}

}  // namespace medimg
