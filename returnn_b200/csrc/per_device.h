// What a process sets up once per device: attributes of a kernel (shared memory beyond 48 KB, clusters of more than 8 CTAs) hold for the device
// that is current when they are set, and a kernel that needs them fails to launch on any other.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>

class RbPerDevice {
  std::atomic<uint64_t> done_{0};
  static uint64_t bit() {  // of the current device; 0: not kept, set up every time
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? (uint64_t)1 << dev : 0;
  }

 public:
  bool needed() const { return !(done_.load(std::memory_order_acquire) & bit()); }
  void done() { done_.fetch_or(bit(), std::memory_order_release); }
};
