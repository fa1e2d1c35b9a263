// Launchers for the PLAIN kernels and the arithmetic self-test.
#include "kernels/bvh2.cuh"
#include "kernels/plain.cuh"
#include "launch.hpp"

namespace rtl {

namespace {
constexpr uint32_t PLAIN_BLOCK = 128;

__global__ void k_selftest(uint32_t* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  volatile float pz = 0.0f, nz = -0.0f, three = 3.0f, two = 2.0f, tiny = 5.877471754e-39f;  // 2^-127, subnormal
  out[0] = __float_as_uint(fminf(nz, pz));
  out[1] = __float_as_uint(fminf(pz, nz));
  out[2] = __float_as_uint(fmaxf(nz, pz));
  out[3] = __float_as_uint(fmaxf(pz, nz));
  out[4] = __float_as_uint(__frcp_rn(three));
  out[5] = __float_as_uint(__fsqrt_rn(two));
  out[6] = __float_as_uint(__frcp_rn(tiny));  // subnormal operand: no flush to zero
  out[7] = __float_as_uint(__fdiv_rn(1.0f, three));
  out[8] = __float_as_uint(__fmul_rn(tiny, 1.0f));
  for (int k = 9; k < 16; ++k) out[k] = 0;
}

// Lanes of a warp that take rays (a power of two). A launch of few rays is bound by the longest of
// each warp's chains of loads, which the lanes of a warp lengthen for one another, so its rays are
// spread over warps, down to one each, while those stay below 32 an SM. 4,096 visibility rays over
// 900 boxes 39.1 -> 16.3 us, 300 34.6 -> 11.7, 10,000 GI rays over 100k triangles 202 -> 147 (with
// 16 or 64 warps an SM 151 and 160); from 300,000 rays on the warps are full.
uint32_t plain_width(uint32_t n) {
  uint32_t width = 32;
  while (width > 1 && n < width * (148u * 32u)) width /= 2;
  return width;
}
template <class K, class Src>
cudaError_t run_plain(K kernel, const SceneView& s, const Src& src, uint32_t n, rtk::DevStatus* st, cudaStream_t stream) {
  const uint32_t width = plain_width(n), per_block = PLAIN_BLOCK / 32 * width;
  kernel<<<(uint32_t)(((uint64_t)n + per_block - 1) / per_block), PLAIN_BLOCK, 0, stream>>>(s.words, src, n, width, st);
  return cudaGetLastError();
}
template <class Src>
cudaError_t launch_plain_of(const SceneView& s, uint32_t mode, const Src& src, uint32_t n, rtk::DevStatus* st,
                            cudaStream_t stream) {
  if (s.layout == 0)
    return mode == 0 ? run_plain(rtk::k_gi_plain<0, Src>, s, src, n, st, stream) : run_plain(rtk::k_gi_plain<1, Src>, s, src, n, st, stream);
  return mode == 0 ? run_plain(rtk::k_rs_plain<0, Src>, s, src, n, st, stream) : run_plain(rtk::k_rs_plain<1, Src>, s, src, n, st, stream);
}
}  // namespace

cudaError_t launch_plain(const SceneView& s, uint32_t mode, const float4* rays, void* hits, uint32_t n,
                         rtk::DevStatus* st, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (s.layout != 2) return launch_plain_of(s, mode, rtk::OneBatch{rays, nullptr, hits}, n, st, stream);
  const dim3 grid((n + PLAIN_BLOCK - 1) / PLAIN_BLOCK), block(PLAIN_BLOCK);
  if (mode == 0) rtk::k_rs2_plain<false><<<grid, block, 0, stream>>>(s.words, rays, hits, n, st);
  else rtk::k_rs2_plain<true><<<grid, block, 0, stream>>>(s.words, rays, hits, n, st);
  return cudaGetLastError();
}

cudaError_t launch_plain_split(const SceneView& s, uint32_t mode, const rtk::SplitRays& src, uint32_t n, rtk::DevStatus* st,
                               cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (s.layout == 2) return cudaErrorInvalidValue;
  return launch_plain_of(s, mode, src, n, st, stream);
}

cudaError_t launch_selftest(uint32_t* out16, cudaStream_t stream) {
  k_selftest<<<1, 32, 0, stream>>>(out16);
  return cudaGetLastError();
}

}  // namespace rtl
