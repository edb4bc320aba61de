// Number of SMs of the current device, asked once per device.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace adb200 {

inline int sm_count() {
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices];                 // 0: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 148;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    known[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace adb200
