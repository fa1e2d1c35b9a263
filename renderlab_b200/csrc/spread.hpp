// How many warps of a kernel the current device holds, and how a launch's rays are spread over them.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <mutex>

namespace rtl {

// Resident blocks of `kernel` on the current device, cached per (kernel, device) under a lock:
// kernels of one signature share this template instance but can differ in registers and shared
// memory, and rt_trace_static calls arrive from any thread without a context lock.
template <class K>
cudaError_t resident_blocks(K kernel, int block, uint32_t& out) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, uint32_t> cached;
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cached.find(key);
    if (it != cached.end()) {
      out = it->second;
      return cudaSuccess;
    }
  }
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0)) != cudaSuccess) return e;
  out = (uint32_t)sms * (uint32_t)(per_sm > 0 ? per_sm : 1);
  std::lock_guard<std::mutex> lock(mu);
  cached[key] = out;
  return cudaSuccess;
}

// Lanes of a warp that take rays: the least power of two at which `warps` warps hold n rays (32 where none
// does). A launch that does not fill the GPU is bound by its longest rays' chains of loads, and a
// warp's lanes delay one another where they part, so its rays are spread over as many warps as pay.
inline uint32_t spread_width(uint64_t warps, uint32_t n) {
  uint32_t width = 1;
  while (width < 32 && warps * width < n) width *= 2;
  return width;
}

}  // namespace rtl
