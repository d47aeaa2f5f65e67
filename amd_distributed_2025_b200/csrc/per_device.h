// Once per device of the process: settings such as a kernel's opt-in to large shared memory hold for the device that
// was current when they were made, so "once per process" leaves every other device without them.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace b200 {

class OncePerDevice {
 public:
  // Runs `set` unless it has succeeded on the current device before; a failure is returned and tried again by the next
  // call.  (Two threads may both run it the first time: such settings may be made twice.)
  template <typename F>
  cudaError_t operator()(F&& set) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool known = dev >= 0 && dev < kDevices;
    if (known && done_[dev].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t r = set();
    if (known && r == cudaSuccess) done_[dev].store(true, std::memory_order_release);
    return r;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<bool> done_[kDevices] = {};
};

// The two opt-ins of a cluster kernel.
template <typename K>
cudaError_t opt_in(K kernel, int smem, bool large_clusters) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess || !large_clusters) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

}  // namespace b200
