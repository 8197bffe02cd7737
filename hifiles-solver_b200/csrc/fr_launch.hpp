// fr_launch.hpp -- the opt-in to more than 48 KB of dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>

namespace frb {

// Raises a kernel's limit where it needs to, once per device: the limit belongs
// to the kernel on a device, and a process may hold solvers on several.  One
// static object per kernel; threads may share it (the limit is set again at worst).
class SmemLimit {
 public:
  void operator()(const void* kernel, size_t bytes)
  {
    if (bytes <= 48 * 1024) return;
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (set_.load(std::memory_order_acquire) & bit) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
      set_.fetch_or(bit, std::memory_order_release);
  }

 private:
  std::atomic<unsigned long long> set_{0};
};

}  // namespace frb
