// smem_limit.h -- kernels that take more dynamic shared memory than the 48 KB
// every kernel may.
#pragma once
#include <atomic>
#include <cstddef>
#include <cuda_runtime.h>

namespace dmsc {

// The limit belongs to a kernel on one device, and contexts of one process may
// be on several.  So it is raised once per device (a static object beside the
// launch): the first call on a device sets it, later ones look at a bit.  Two
// threads that come first together both set it, to the same value.
class SmemLimit {
  std::atomic<unsigned long long> done{0};  // a bit per device (a device past 63: set by every call)

 public:
  // `bytes` for the kernels, on the current device
  template <typename... K>
  cudaError_t raise(size_t bytes, K... kernels) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (e != cudaSuccess || (done.load(std::memory_order_acquire) & bit)) return e;
    ((e = e == cudaSuccess ? cudaFuncSetAttribute(kernels, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) : e), ...);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

}  // namespace dmsc
