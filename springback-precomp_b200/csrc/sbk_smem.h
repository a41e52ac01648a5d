// The dynamic shared memory a kernel may be launched with.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace sbk {

// One per kernel (a static of the function that launches it). allow() raises
// the kernel's limit to all that a block may have, once per device: never to
// the size of the launch at hand, for that would lower the limit under
// another thread that is about to launch a larger one. Every thread sets the
// same value, so it does not matter who comes first. Later launches, those
// inside a stream capture among them, make no attribute call.
class SmemLimit {
 public:
  template <class K>
  cudaError_t allow(K kern) {
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const bool known = dev >= 0 && dev < kDevices;
    if (known && done_[dev].load(std::memory_order_acquire)) return cudaSuccess;
    int most = 0;
    cudaFuncAttributes own;
    if ((err = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return err;
    if ((err = cudaFuncGetAttributes(&own, kern)) != cudaSuccess) return err;
    err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               most - static_cast<int>(own.sharedSizeBytes));
    if (err == cudaSuccess && known) done_[dev].store(true, std::memory_order_release);
    return err;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<bool> done_[kDevices] = {};
};

}  // namespace sbk
