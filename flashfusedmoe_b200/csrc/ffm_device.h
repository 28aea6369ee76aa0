// Values the host side finds out once for every device: function attributes and occupancy belong to a device, and one
// process may launch on several.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>

namespace ffm {

constexpr int MAX_DEVICES = 64;

// Positive integers by device, 0 where not known yet. Threads may race to the first call: each finds the same value.
struct PerDevice {
  std::atomic<int> value[MAX_DEVICES] = {};

  // the current device's value, from `find` at the first call on it; what `find` returns is kept if positive
  template <typename F>
  int get(F&& find) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return find();
    int v = value[dev].load(std::memory_order_acquire);
    if (v <= 0) {
      v = find();
      if (v > 0) value[dev].store(v, std::memory_order_release);
    }
    return v;
  }
};

}  // namespace ffm
