// Launchers for the PLAIN kernels over the GI layout.
#include "plain_run.hpp"

namespace rtl {

namespace {
// GI closest hits have a second kernel of PLAIN_FEW_BLOCKS blocks an SM, whose registers hold all (none
// spilled). It takes the launches whose warps it holds at once, at the other kernel's width or with at
// least 16 rays a warp: 60,000 rays over 500 instances 1,787 us against 1,869, 90,000 2,115 against
// 2,222, 20,000 camera rays 596 against 627. In a second wave it loses (130,000: 3,187 against 2,695).
template <class Src>
cudaError_t run_gi_closest(const SceneView& s, const Src& src, uint32_t n, rtk::DevStatus* st, cudaStream_t stream) {
  const auto many = rtk::k_gi_plain<0, Src, rtk::PLAIN_MIN_BLOCKS>, few = rtk::k_gi_plain<0, Src, rtk::PLAIN_FEW_BLOCKS>;
  uint32_t full = 0, full_few = 0;
  cudaError_t e = resident_blocks(many, PLAIN_BLOCK, full);
  if (e == cudaSuccess) e = resident_blocks(few, PLAIN_BLOCK, full_few);
  if (e != cudaSuccess) return e;
  const uint64_t warps = (uint64_t)full * (PLAIN_BLOCK / 32), warps_few = (uint64_t)full_few * (PLAIN_BLOCK / 32);
  const uint32_t width = plain_width(warps, n), width_few = spread_width(warps_few, n);
  if (n <= warps_few * width_few && (width_few == width || width_few >= 16))
    return run_plain_at(few, width_few, s, src, n, st, stream);
  return run_plain_at(many, width, s, src, n, st, stream);
}
// GI any hits: with less than 16 rays a warp, the walk by shared steps (see gi_blocked).
template <class Src>
cudaError_t run_gi_any(const SceneView& s, const Src& src, uint32_t n, rtk::DevStatus* st, cudaStream_t stream) {
  const auto full_warps = rtk::k_gi_plain<1, Src, rtk::PLAIN_ANY_BLOCKS, false>;
  uint32_t full = 0;
  const cudaError_t e = resident_blocks(full_warps, PLAIN_BLOCK, full);
  if (e != cudaSuccess) return e;
  const uint32_t width = plain_width((uint64_t)full * (PLAIN_BLOCK / 32), n);
  if (width < 16) return run_plain_at(rtk::k_gi_plain<1, Src, rtk::PLAIN_ANY_BLOCKS, true>, width, s, src, n, st, stream);
  return run_plain_at(full_warps, width, s, src, n, st, stream);
}
}  // namespace

template <class Src>
cudaError_t launch_plain_gi(const SceneView& s, uint32_t mode, const Src& src, uint32_t n, rtk::DevStatus* st,
                            cudaStream_t stream) {
  return mode == 0 ? run_gi_closest(s, src, n, st, stream) : run_gi_any(s, src, n, st, stream);
}
template cudaError_t launch_plain_gi(const SceneView&, uint32_t, const rtk::OneBatch&, uint32_t, rtk::DevStatus*, cudaStream_t);
template cudaError_t launch_plain_gi(const SceneView&, uint32_t, const rtk::SplitRays&, uint32_t, rtk::DevStatus*, cudaStream_t);

}  // namespace rtl
