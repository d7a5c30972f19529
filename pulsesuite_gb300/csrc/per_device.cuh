// What a process asks or sets once for each device it uses.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace sbe {

constexpr int kDevices = 64;   // devices remembered; a later one is asked every time

// multiprocessors of the current device (1 when it cannot say)
inline int sm_count() {
  static std::atomic<int> known[kDevices];
  int dev = -1, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  if (dev < kDevices && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
    return 1;
  if (dev < kDevices) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

// The dynamic shared memory limit of kernel K raised to bytes (the same in every call) on the
// current device: the limit belongs to the device's copy of the kernel.  A failure is returned and
// not remembered.
template <auto K>
inline cudaError_t raise_smem(int bytes) {
  static std::atomic<unsigned long long> raised{0};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < kDevices ? 1ull << dev : 0;
  if (raised.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) raised.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

}  // namespace sbe
