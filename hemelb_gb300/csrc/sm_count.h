// Multiprocessors of the current device.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>

namespace hlbg {

// What the launch rules were measured on, and the answer where the device gives none.
constexpr int kMeasuredSms = 152;

// Asked once per device (a launch asks every time).
inline int sm_count() {
  static std::atomic<int> known[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return kMeasuredSms;
  if (dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return kMeasuredSms;
  if (dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace hlbg
