// Launches of the PLAIN kernels: the rays of a launch spread over warps. The GI kernels are compiled apart
// from the others (kernels_plain_gi.cu): with both layouts' kernels in one unit the compiler spilled 120
// bytes in the reflection any-hit kernel instead of 60 (1M rays over 500 instances 7.65 against 6.00 ms).
#pragma once
#include "kernels/plain.cuh"
#include "launch.hpp"
#include "spread.hpp"

namespace rtl {

constexpr uint32_t PLAIN_BLOCK = 128;

// A launch at `width` rays a warp.
template <class K, class Src>
cudaError_t run_plain_at(K kernel, uint32_t width, const SceneView& s, const Src& src, uint32_t n, rtk::DevStatus* st,
                         cudaStream_t stream) {
  const uint32_t per_block = PLAIN_BLOCK / 32 * width;
  kernel<<<(uint32_t)(((uint64_t)n + per_block - 1) / per_block), PLAIN_BLOCK, 0, stream>>>(s.words, src, n, width, st);
  return cudaGetLastError();
}
// Rays are spread over the resident warps (spread_width). 4,096 visibility rays over 900 boxes 39.1 -> 16.3
// us, 10,000 GI rays over 500 instances 1,441 -> 859 us (GI layout); more warps than are resident cost
// waves of nearly idle warps: 60,000 there 1,855 us with 32 rays a warp, 1,949 with 16, 2,329 with 8; over
// 20 listed instances 385, 407 and 495 us. One ray a warp pays up to a quarter past them, where the last
// rays take the place of the first to end: 5,000 over one mesh 84 us, 113 with two.
inline uint32_t plain_width(uint64_t warps, uint32_t n) { return 4 * (uint64_t)n <= 5 * warps ? 1 : spread_width(warps, n); }
template <class K, class Src>
cudaError_t run_plain(K kernel, const SceneView& s, const Src& src, uint32_t n, rtk::DevStatus* st, cudaStream_t stream) {
  uint32_t full = 0;
  const cudaError_t e = resident_blocks(kernel, PLAIN_BLOCK, full);
  if (e != cudaSuccess) return e;
  return run_plain_at(kernel, plain_width((uint64_t)full * (PLAIN_BLOCK / 32), n), s, src, n, st, stream);
}

// The GI layout's launches (instantiated for the two ray sources in kernels_plain_gi.cu).
template <class Src>
cudaError_t launch_plain_gi(const SceneView& s, uint32_t mode, const Src& src, uint32_t n, rtk::DevStatus* st,
                            cudaStream_t stream);

}  // namespace rtl
