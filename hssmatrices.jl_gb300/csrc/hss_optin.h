// The opt-in to more than 48 KB of dynamic shared memory of a kernel.  The attribute
// belongs to the kernel on one device, so it is set once for each device that launches
// the kernel; an attempt that failed is made again.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace hss {

// One per kernel (a function's static object).
class SmemOptIn {
 public:
  // `kernel` may take `bytes` (always the same) on the current device from here on.
  cudaError_t operator()(const void* kernel, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t(1) << dev : 0;
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};   // a bit per device; devices beyond 63 set it each time
};

}  // namespace hss
