// Values the host side finds out once for every device: function attributes and occupancy belong to a device, and one
// process may launch on several.
#pragma once

#include <cuda_runtime.h>

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

// Set by the layer driver (ffm_layer.cu) for the launches of this host thread that directly follow a kernel of this library
// on their stream: they may be placed on the GPU while that kernel runs out (see chain_wait in ffm_common.cuh).
inline thread_local bool follows_kernel = false;

// Launch with up to two attributes: a cluster of `cluster` CTAs (0: none), and placement ahead of the end of the kernel
// before it on the stream. Only for kernels that begin with chain_wait().
template <typename... P, typename... A>
bool launch_kernel(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool chained, int cluster,
                   const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 0) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  if (cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

}  // namespace ffm
