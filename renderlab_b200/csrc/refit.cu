// GPU refit of one BLAS of an uploaded scene (near_field::refit_bvh, near_field.rs:445-478, on the
// device): new positions for the same vertices, the BVH4-Q8 node boxes recomputed bottom-up and
// quantised with the host quantiser's exact arithmetic (quantize_node, near_field.rs:481-525), so
// the words equal those of rt_blas_refit followed by packing, bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cfloat>
#include <cmath>
#include <vector>

#include "ctx.hpp"
#include "kernels/bvh4_quant.cuh"
#include "kernels/common.cuh"

using namespace rtc;

namespace {

using namespace rtq;

// GI: the new positions into the BLAS's position words.
__global__ void k_refit_positions(uint32_t* __restrict__ dst, const float* __restrict__ pos, uint32_t n_floats) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_floats) dst[i] = __float_as_uint(pos[i]);
}

// Reflection: each packed triangle's a, b - a, c - a from its primitive's vertices (the packer's
// arithmetic: one f32 subtraction a component).
__global__ void k_refit_triangles(View v, uint32_t n_tris) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tris) return;
  uint32_t* x = v.w + v.tris + 12 * (size_t)t;
  const uint32_t prim = x[9];
  const float* a = v.pos + 3 * (size_t)v.src[3 * (size_t)prim];
  const float* b = v.pos + 3 * (size_t)v.src[3 * (size_t)prim + 1];
  const float* c = v.pos + 3 * (size_t)v.src[3 * (size_t)prim + 2];
  for (int j = 0; j < 3; ++j) {
    x[j] = __float_as_uint(a[j]);
    x[3 + j] = __float_as_uint(__fsub_rn(b[j], a[j]));
    x[6 + j] = __float_as_uint(__fsub_rn(c[j], a[j]));
  }
}

// The words of a record that say where its BLAS's nodes, leaves, positions and indices (GI) or nodes and
// triangles (reflection) lie; `r`: words 18 on.
std::array<uint32_t, 4> blas_of(bool gi, const uint32_t* r) {
  if (gi) return {r[0], r[1], r[2], r[3]};
  return {r[0] & ~3u, r[1] & ~3u, 0u, 0u};
}

// Whether a leaf that no instance's root reaches lies inside the scene's words, as the upload's
// admission checks those that one does (`words`: the scene's, read for the GI layout alone).
bool leaf_inside(const rt_scene* scene, const uint32_t* rec, uint32_t c, const std::vector<uint32_t>& words) {
  const size_t n = scene->n_words;
  if (scene->layout != 0) return (rec[19] & ~3u) + 12 * ((size_t)((c & ~LEAF) >> 4) + (c & 15u)) <= n;
  const size_t l = rec[19] + 2 * (size_t)(c & ~LEAF);
  if (l + 2 > n) return false;
  const size_t first = rec[21] + (size_t)words[l], count = words[l + 1];
  if (first + count > n) return false;
  for (size_t k = first; k < first + count; ++k)
    if (rec[20] + 3 * (size_t)words[k] + 3 > n) return false;
  return true;
}

// The BLAS's topology (once per BLAS): what the refit's launches need, triangle / position counts.
// Every node up to the highest root that an instance enters the BLAS at is refit, as the host's
// refit does, reached from a root or not (a file of several levels holds such nodes, and other
// instances may enter at them).
rt_status levels_of(rt_ctx* ctx, rt_scene* scene, const uint32_t* rec, RefitLevels& out) {
  const bool gi = scene->layout == 0;
  const size_t nodes = gi ? rec[18] : (rec[18] & ~3u);
  uint32_t n = 0, tris = 0;
  for (size_t i = 0; i < scene->info.instances; ++i) {
    const uint32_t* r = scene->blas_words.data() + 6 * i;
    const uint32_t root = gi ? r[4] : r[2];
    if (blas_of(gi, r) != blas_of(gi, rec + 18) || root == EMPTY) continue;
    if (!(root & LEAF)) n = std::max(n, root + 1);  // postorder: the root is the last node
    else if (!gi) tris = std::max(tris, ((root & ~LEAF) >> 4) + (root & 15u));  // a single leaf: its triangles alone
  }
  out.node_count = n;
  out.tri_count = tris;
  if (gi) {  // the packer lays a mesh's positions (3 words each) right before its indices
    if (rec[21] < rec[20] || (rec[21] - rec[20]) % 3 != 0) return fail(ctx, RT_ERR_LAYOUT, "refit: GI position words");
    out.position_count = (rec[21] - rec[20]) / 3;
  }
  if (n == 0) return RT_OK;
  std::vector<uint32_t> w(16 * (size_t)n);
  RT_CUDA(ctx, wait_changes(scene));
  RT_CUDA(ctx, cudaMemcpy(w.data(), scene->d_words + nodes, w.size() * 4, cudaMemcpyDeviceToHost));
  for (uint32_t k = 0; k < n; ++k)
    for (int s = 0; s < 4; ++s) {
      const uint32_t c = w[16 * (size_t)k + 6 + s];
      if (c != EMPTY && !(c & LEAF) && c >= k) return fail(ctx, RT_ERR_LAYOUT, "refit: BLAS children must precede their parent");
    }
  // the tree from the last root: each node's parent and inner children
  std::vector<uint32_t> parent(n, EMPTY);
  std::vector<uint8_t> inner(n, rtq::NEVER);
  inner[n - 1] = 0;
  for (uint32_t k = n; k-- > 0;) {
    if (inner[k] == rtq::NEVER) continue;
    for (int s = 0; s < 4; ++s) {
      const uint32_t c = w[16 * (size_t)k + 6 + s];
      if (c == EMPTY || (c & LEAF)) continue;
      parent[c] = k, inner[c] = 0, ++inner[k];
    }
  }
  const bool tree = std::find(inner.begin(), inner.end(), rtq::NEVER) == inner.end();
  std::vector<uint32_t> words, height(tree ? 0 : n, 0), order;
  if (!tree && gi) {
    words.resize(scene->n_words);
    RT_CUDA(ctx, cudaMemcpy(words.data(), scene->d_words, 4 * words.size(), cudaMemcpyDeviceToHost));
  }
  uint32_t top = 0;
  for (uint32_t k = 0; k < n; ++k) {
    uint32_t h = 1, most = 0;
    for (int s = 0; s < 4; ++s) {
      const uint32_t c = w[16 * (size_t)k + 6 + s];
      if (c == EMPTY) continue;
      if (c & LEAF) {
        if (!gi) most = std::max(most, ((c & ~LEAF) >> 4) + (c & 15u));
        if (!tree && inner[k] == rtq::NEVER && !leaf_inside(scene, rec, c, words)) h = 0;
      } else if (!tree) {
        h = h && height[c] ? std::max(h, height[c] + 1) : 0;
      }
    }
    if (h == 0) continue;  // leaves outside the words below it: no ray enters here, and it stays as it is
    tris = std::max(tris, most);
    if (!tree) height[k] = h, top = std::max(top, h);
  }
  out.tri_count = tris;
  if (!tree) {
    std::vector<uint32_t>& start = out.level_start;  // height h + 1 at start[h] on
    start.assign(top + 1, 0);
    for (uint32_t h : height)
      if (h) ++start[h];
    for (uint32_t h = 1; h <= top; ++h) start[h] += start[h - 1];
    order.resize(start[top]);
    std::vector<uint32_t> next(start.begin(), start.end());
    for (uint32_t k = 0; k < n; ++k)
      if (height[k]) order[next[height[k] - 1]++] = k;
  }
  // one allocation: parents, counters of a launch, inner child counts; or the order
  if (device_alloc(ctx, &out.d_tree, tree ? 9 * (size_t)n : 4 * std::max<size_t>(order.size(), 1), true) != cudaSuccess) {
    cudaGetLastError();
    out.d_tree = nullptr;
    return fail(ctx, RT_ERR_OOM, "refit tree");
  }
  cudaError_t e = tree ? cudaMemcpy(out.d_tree, parent.data(), 4 * (size_t)n, cudaMemcpyHostToDevice)
                       : cudaMemcpy(out.d_tree, order.data(), 4 * order.size(), cudaMemcpyHostToDevice);
  if (tree && e == cudaSuccess) e = cudaMemcpy(out.d_tree + 2 * (size_t)n, inner.data(), n, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(out.d_tree);
    out.d_tree = nullptr;
    return fail(ctx, RT_ERR_CUDA, "refit tree: %s", cudaGetErrorString(e));
  }
  return RT_OK;
}

}  // namespace

rt_status rt_scene_refit(rt_ctx* ctx, rt_scene* scene, uint32_t instance, const float* d_positions,
                         uint32_t n_positions, const uint32_t* d_indices, uint32_t n_indices, void* stream) {
  if (!ctx || !scene || !d_positions) return fail(ctx, RT_ERR_INVALID_ARG, "null argument");
  if (instance >= scene->info.instances) return fail(ctx, RT_ERR_INVALID_ARG, "no instance %u", instance);
  if (scene->layout == RT_LAYOUT_REFLECTION_BVH2)
    return fail(ctx, RT_ERR_UNSUPPORTED, "refit covers the BVH4 layouts (the legacy BVH2 one is rebuilt on the host)");
  const bool gi = scene->layout == 0;
  if (!gi && !d_indices) return fail(ctx, RT_ERR_INVALID_ARG, "the reflection layout refits from the triangle list");
  std::lock_guard<std::mutex> lock(ctx->mu);
  RT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  RT_CUDA(ctx, cudaStreamIsCapturing(s, &capture));
  uint32_t rec[24] = {};
  std::copy_n(scene->blas_words.begin() + 6 * (size_t)instance, 6, rec + 18);
  if (capture != cudaStreamCaptureStatusNone)  // refused where the capture allows no synchronous call
    RT_CUDA(ctx, cudaMemcpy(rec, scene->d_words + (gi ? 16 + 32 * (size_t)instance : 8 + 24 * (size_t)instance), sizeof rec,
                            cudaMemcpyDeviceToHost));
  const uint32_t base = gi ? rec[18] : (rec[18] & ~3u);
  const std::array<uint32_t, 4> key = blas_of(gi, rec + 18);
  auto it = scene->refit.find(key);
  if (it == scene->refit.end()) {
    RefitLevels lv;
    rt_status st = levels_of(ctx, scene, rec, lv);
    if (st != RT_OK) return st;
    it = scene->refit.emplace(key, std::move(lv)).first;
  }
  const RefitLevels& lv = it->second;
  if (gi && n_positions != lv.position_count)
    return fail(ctx, RT_ERR_INVALID_ARG, "the BLAS has %u positions, not %u", lv.position_count, n_positions);
  if (!gi && (size_t)n_indices < 3 * (size_t)lv.tri_count)
    return fail(ctx, RT_ERR_INVALID_ARG, "the triangle list is shorter than the BLAS's triangles");
  if (scene->d_wide8) {  // the derived 8-wide layout no longer matches: rt_scene_prepare again
    RT_CUDA(ctx, cudaFree(scene->d_wide8));
    scene->d_wide8 = nullptr;
    scene->device_bytes -= scene->wide8_bytes;
    ctx->scene_bytes -= scene->wide8_bytes;
    scene->wide8_bytes = 0;
  }
  Change change(scene, s);
  if (capture == cudaStreamCaptureStatusNone) RT_CUDA(ctx, change.start());  // a captured refit is the replay's caller's to order
  View v{};
  v.w = scene->d_words;
  v.layout = scene->layout;
  v.nodes = base;
  if (gi) {
    v.leaves = rec[19], v.positions = rec[20], v.indices = rec[21];
    const uint32_t nf = 3 * n_positions;
    if (nf) k_refit_positions<<<(nf + 255) / 256, 256, 0, s>>>(scene->d_words + v.positions, d_positions, nf);
  } else {
    v.tris = rec[19] & ~3u, v.pos = d_positions, v.src = d_indices;
    if (lv.tri_count) k_refit_triangles<<<(lv.tri_count + 255) / 256, 256, 0, s>>>(v, lv.tri_count);
  }
  RT_CUDA(ctx, cudaGetLastError());
  const auto blocks = [](uint64_t nodes) { return (uint32_t)((4 * nodes + REFIT_BLOCK - 1) / REFIT_BLOCK); };
  for (size_t h = 0; h + 1 < lv.level_start.size(); ++h) {
    const uint32_t first = lv.level_start[h], n = lv.level_start[h + 1] - first;
    if (n) k_refit_level<REFIT_BLOCK><<<blocks(n), REFIT_BLOCK, 0, s>>>(v, lv.d_tree + first, n);
  }
  if (lv.node_count && lv.level_start.empty()) {
    const uint32_t n = lv.node_count;
    RT_CUDA(ctx, cudaMemsetAsync(lv.d_tree + n, 0, 4 * (size_t)n, s));
    k_refit_up<REFIT_BLOCK><<<blocks(n), REFIT_BLOCK, 0, s>>>(
        v, n, lv.d_tree, reinterpret_cast<const uint8_t*>(lv.d_tree + 2 * (size_t)n), lv.d_tree + n);
  }
  RT_CUDA(ctx, cudaGetLastError());
  return RT_OK;
}

rt_status rt_scene_read_words(rt_ctx* ctx, const rt_scene* scene, size_t first, size_t n, uint32_t* out) {
  if (!ctx || !scene || (n && !out)) return fail(ctx, RT_ERR_INVALID_ARG, "null argument");
  if (first > scene->n_words || n > scene->n_words - first) return fail(ctx, RT_ERR_INVALID_ARG, "words out of range");
  RT_CUDA(ctx, cudaSetDevice(ctx->device));
  RT_CUDA(ctx, wait_changes(scene));
  if (n) RT_CUDA(ctx, cudaMemcpy(out, scene->d_words + first, n * 4, cudaMemcpyDeviceToHost));
  return RT_OK;
}
