// Launchers for the PLAIN kernels over the reflection layouts and the arithmetic self-test.
#include "kernels/bvh2.cuh"
#include "plain_run.hpp"

namespace rtl {

namespace {
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

template <class Src>
cudaError_t launch_plain_of(const SceneView& s, uint32_t mode, const Src& src, uint32_t n, rtk::DevStatus* st,
                            cudaStream_t stream) {
  if (s.layout == 0) return launch_plain_gi(s, mode, src, n, st, stream);
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
