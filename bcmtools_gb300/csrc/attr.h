// attr.h -- kernel attributes, set once per kernel and device.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

namespace bcmg {

// One per kernel (a static of its launcher).  A function attribute holds for the
// device that is current when it is set, and a process may have contexts on
// several, so the flag is one bit per device; two threads that both find it clear
// set the same values.  Not a stream operation: allowed during a capture.
class SharedMemory {
 public:
  template <class K>
  cudaError_t allow(K kern, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? uint64_t{1} << dev : 0;  // further ones: on every launch
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

// CTAs of a kernel that the current device holds at once, asked for once per
// device.
class Resident {
 public:
  template <class K>
  cudaError_t ctas(K kern, int threads, size_t bytes, int* out) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && (*out = n_[dev].load(std::memory_order_relaxed)) > 0) return cudaSuccess;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kern, threads, bytes);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    *out = sms * per_sm;
    if (dev < 64) n_[dev].store(*out, std::memory_order_relaxed);
    return cudaSuccess;
  }

 private:
  std::atomic<int> n_[64] = {};
};

}  // namespace bcmg
