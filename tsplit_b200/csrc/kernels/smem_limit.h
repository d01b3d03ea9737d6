// Dynamic shared memory above 48 KB: allowed per kernel AND device, so "already raised" is remembered per device (a bit
// each; a device past the 64th is raised every time).  One object per kernel, as a function-local static beside its
// launch.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace tsb_launch {

class SmemLimit {
 public:
  template <class K>
  cudaError_t raise(K* kernel, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (raised_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) raised_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<unsigned long long> raised_{0};
};

}  // namespace tsb_launch
