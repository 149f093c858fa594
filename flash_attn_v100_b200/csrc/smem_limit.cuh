// Dynamic shared memory a kernel may ask for, raised once per device and size instead of before every launch.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

namespace fa {

// One per kernel (a function-local static beside its launch).  The call it saves was most of the 2.6 us by which a decode launch from C
// became shorter (8.1 to 5.5 us).
struct SharedMemoryLimit {
  std::atomic<int> bytes[64] = {};
  std::mutex mu;
  cudaError_t raise(const void* kernel, int need) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, need);
    if (bytes[dev].load(std::memory_order_acquire) >= need) return cudaSuccess;
    std::lock_guard<std::mutex> lock(mu);          // (a smaller size set last would undo a larger one)
    if (bytes[dev].load(std::memory_order_relaxed) >= need) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, need);
    if (e == cudaSuccess) bytes[dev].store(need, std::memory_order_release);
    return e;
  }
};

}  // namespace fa
