// smem_optin.h -- a kernel's opt-in to more than 48 KB of dynamic shared
// memory.  cudaFuncSetAttribute holds for the current device alone, so what was
// granted is kept for each device; a call that failed is made again.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <mutex>

namespace medimg {

class SmemOptIn {
 public:
  // get_device(&dev) names the current device, raise(bytes) makes the call;
  // each returns a cudaError_t.  Every kernel has 48 KB without one.
  template <typename GetDevice, typename Raise>
  cudaError_t ensure(size_t bytes, GetDevice &&get_device, Raise &&raise) {
    if (bytes <= kFree) return cudaSuccess;
    int dev = 0;
    cudaError_t e = get_device(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kDevices) return raise(bytes);
    std::lock_guard<std::mutex> lock(mu_);
    if (bytes <= granted_[dev]) return cudaSuccess;
    if ((e = raise(bytes)) == cudaSuccess) granted_[dev] = bytes;
    return e;
  }

 private:
  static constexpr size_t kFree = 48 * 1024;
  static constexpr int kDevices = 64;
  std::mutex mu_;
  size_t granted_[kDevices] = {};
};

}  // namespace medimg
