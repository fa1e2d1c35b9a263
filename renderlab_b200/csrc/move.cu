// Moving the instances of an uploaded scene on the device: the records' rows and world boxes
// (the packers' arithmetic: gi_bvh.rs:230-274, reflection_software.rs:347-388), the top level
// refit over the new boxes as instance_bvh::place does for a moved set (instance_bvh.rs:162-275:
// refit, word 3 counting refits, a rebuild after 64, made on the device by tlas_build.cu), and
// the reflection layout's scene bounds
// (reflection_software.rs:295-313). Every float operation is an explicit round-to-nearest step in
// the host code's order, so the words equal rt_move_instances_host's, bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ctx.hpp"
#include "kernels/common.cuh"

using namespace rtc;

namespace {

using rtk::EMPTY;
using rtk::LEAF;

constexpr size_t TOP_WORDS = 32;  // a top-level node: 24 box words, 4 child ids, 4 unused

struct Box {
  float lo[3], hi[3];
};

__device__ __forceinline__ float lo_of(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float hi_of(float a, float b) { return b > a ? b : a; }
__device__ __forceinline__ Box empty_box() { return Box{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}}; }
__device__ __forceinline__ void grow(Box& b, const float* l, const float* h) {
  for (int a = 0; a < 3; ++a) b.lo[a] = lo_of(b.lo[a], l[a]), b.hi[a] = hi_of(b.hi[a], h[a]);
}

// pack.cpp's instance_box: the eight corners of the object box through the model (x, + y, + z,
// + w, rounded in turn), then the layout's margin.
__device__ Box instance_box(uint32_t layout, const float* m, const float* obj) {
  Box wb = empty_box();
  for (int c = 0; c < 8; ++c) {
    float p[3], w[3];
    for (int a = 0; a < 3; ++a) p[a] = (c >> a) & 1 ? obj[3 + a] : obj[a];
    for (int r = 0; r < 3; ++r) {
      float acc = __fmul_rn(m[4 * r], p[0]);
      acc = __fadd_rn(__fmul_rn(m[4 * r + 1], p[1]), acc);
      acc = __fadd_rn(__fmul_rn(m[4 * r + 2], p[2]), acc);
      w[r] = __fadd_rn(m[4 * r + 3], acc);
    }
    grow(wb, w, w);
  }
  Box out;
  if (layout == 0) {
    for (int a = 0; a < 3; ++a) {
      const float pad = __fmul_rn(1e-5f, __fadd_rn(1.0f, hi_of(fabsf(wb.lo[a]), fabsf(wb.hi[a]))));
      out.lo[a] = __fsub_rn(wb.lo[a], pad), out.hi[a] = __fadd_rn(wb.hi[a], pad);
    }
    return out;
  }
  float margin = 0.0f;
  for (int a = 0; a < 3; ++a)
    margin = hi_of(margin, hi_of(hi_of(fabsf(wb.hi[a]), fabsf(wb.lo[a])), __fsub_rn(wb.hi[a], wb.lo[a])));
  margin = __fmul_rn(margin, 1e-5f);
  for (int a = 0; a < 3; ++a) out.lo[a] = __fsub_rn(wb.lo[a], margin), out.hi[a] = __fadd_rn(wb.hi[a], margin);
  return out;
}

__global__ void k_move_records(uint32_t* __restrict__ w, uint32_t layout, const rt_instance* __restrict__ moved, uint32_t n,
                               const float* __restrict__ mesh_boxes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const rt_instance& g = moved[i];
  uint32_t* r = w + (layout == 0 ? 16 + 32 * (size_t)i : 8 + 24 * (size_t)i);
  for (int k = 0; k < 12; ++k) r[k] = __float_as_uint(g.rows[k]);
  const Box b = instance_box(layout, g.model, mesh_boxes + 6 * (size_t)g.mesh);
  for (int a = 0; a < 3; ++a) r[12 + a] = __float_as_uint(b.lo[a]), r[15 + a] = __float_as_uint(b.hi[a]);
}

constexpr uint8_t NEVER = 0xff;  // inner children of a node that is not refit

// The top level refit over the records' boxes in one launch: four lanes a node, a child each, climb
// from the nodes without inner children; of a node's inner children the last one done takes the
// node (done[], zeroed before the launch; nothing waits). An inner child's box is grown in slot order
// as instance_bvh::refit_wide does. 2,500 instances, 6 heights: 40 us as a launch per height with a
// thread a node, 16 so (the whole call until the device is done: 144 -> 90 us, 52 of them on the host).
// `refits`: the header's count.
constexpr int TOP_BLOCK = 128;
__global__ void __launch_bounds__(TOP_BLOCK) k_refit_top(uint32_t* __restrict__ w, uint32_t layout, size_t base, uint32_t n,
                                                         const uint32_t* __restrict__ parent,
                                                         const uint8_t* __restrict__ inner, uint32_t* __restrict__ done,
                                                         uint32_t refits) {
  const uint32_t i = (blockIdx.x * TOP_BLOCK + threadIdx.x) / 4;
  if (blockIdx.x == 0 && threadIdx.x == 0) w[3] = refits;
  if (i >= n || inner[i] != 0) return;
  const int c = threadIdx.x & 3;
  const unsigned quad = 0xfu << (threadIdx.x & 28);
  for (uint32_t at = i;;) {
    uint32_t* node = w + base + TOP_WORDS * (size_t)at;
    const uint32_t id = node[24 + c];
    if (id != EMPTY) {
      Box b;
      if (id & LEAF) {
        const uint32_t* r = w + (layout == 0 ? 16 + 32 * (size_t)(id & ~LEAF) : 8 + 24 * (size_t)(id & ~LEAF));
        for (int a = 0; a < 3; ++a) b.lo[a] = __uint_as_float(r[12 + a]), b.hi[a] = __uint_as_float(r[15 + a]);
      } else {  // another thread block may have written it in this launch: past L1
        const uint32_t* child = w + base + TOP_WORDS * (size_t)id;
        uint32_t x[28];
#pragma unroll
        for (int k = 0; k < 28; ++k) x[k] = __ldcg(child + k);
        b = empty_box();
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          if (x[24 + cc] == EMPTY) continue;
          float l[3], h[3];
          for (int a = 0; a < 3; ++a) l[a] = __uint_as_float(x[4 * a + cc]), h[a] = __uint_as_float(x[12 + 4 * a + cc]);
          grow(b, l, h);
        }
      }
      for (int a = 0; a < 3; ++a) node[4 * a + c] = __float_as_uint(b.lo[a]), node[12 + 4 * a + c] = __float_as_uint(b.hi[a]);
    }
    const uint32_t up = parent[at];
    if (up == EMPTY) return;
    __syncwarp(quad);  // the four lanes' words are written
    uint32_t last = 0;
    if (c == 0) {
      __threadfence();
      last = atomicAdd(&done[up], 1u) + 1u == inner[up] ? 1u : 0u;
      __threadfence();
    }
    __syncwarp(quad);  // what lane 0's fence has made visible, the other lanes may read (a shuffle orders no memory)
    if (!__shfl_sync(quad, last, 0, 4)) return;
    at = up;
  }
}

// Parents and inner child counts of a tree built on the device (nodes 0 to n - 1, the root first), and the
// header's refit count, 0 from here.
__global__ void k_top_links(uint32_t* __restrict__ w, size_t base, uint32_t n, uint32_t* __restrict__ parent,
                            uint8_t* __restrict__ inner) {
  const uint32_t* nodes = w + base;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) w[3] = 0;
  if (i >= n) return;
  uint32_t kids = 0;
  for (int c = 0; c < 4; ++c) {
    const uint32_t id = nodes[TOP_WORDS * (size_t)i + 24 + c];
    if (id != EMPTY && !(id & LEAF)) parent[id] = i, ++kids;
  }
  inner[i] = (uint8_t)kids;
  if (i == 0) parent[0] = EMPTY;
}

// The reflection scene bounds: the instances' boxes grown in record order. Each thread grows a
// contiguous run, then the runs are combined in order, neighbours first; a strict comparison keeps
// the earlier of two equal values (+0 and -0), as one sequential pass does.
constexpr int BOUNDS_THREADS = 512;
__global__ void __launch_bounds__(BOUNDS_THREADS) k_scene_bounds(uint32_t* __restrict__ w, uint32_t n) {
  __shared__ Box part[BOUNDS_THREADS / 32];
  const uint32_t t = threadIdx.x, per = (n + BOUNDS_THREADS - 1) / BOUNDS_THREADS;
  Box b = empty_box();
  for (uint32_t i = t * per; i < n && i < (t + 1) * per; ++i) {
    const uint32_t* r = w + 8 + 24 * (size_t)i;
    float l[3], h[3];
    for (int a = 0; a < 3; ++a) l[a] = __uint_as_float(r[12 + a]), h[a] = __uint_as_float(r[15 + a]);
    grow(b, l, h);
  }
  auto combine = [](Box& x, int lanes) {
    for (int off = 1; off < lanes; off *= 2) {
      float l[3], h[3];
      for (int a = 0; a < 3; ++a)
        l[a] = __shfl_down_sync(0xffffffffu, x.lo[a], off), h[a] = __shfl_down_sync(0xffffffffu, x.hi[a], off);
      grow(x, l, h);
    }
  };
  combine(b, 32);
  if ((t & 31) == 0) part[t / 32] = b;
  __syncthreads();
  if (t >= 32) return;
  constexpr int WARPS = BOUNDS_THREADS / 32;
  Box all = t < WARPS ? part[t] : empty_box();
  combine(all, WARPS);
  if (t != 0) return;
  const size_t at = w[4];
  for (int a = 0; a < 3; ++a) w[at + a] = __float_as_uint(all.lo[a]), w[at + 4 + a] = __float_as_uint(all.hi[a]);
}

// Parents and inner child counts of the top level's nodes reachable from the root (the reserve may
// hold unused space: NEVER). Returns how many nodes it has to see: at most those given when it is done.
size_t top_links(const std::vector<uint32_t>& nodes, std::vector<uint32_t>& parent, std::vector<uint8_t>& inner) {
  const size_t nn = nodes.size() / TOP_WORDS;
  size_t need = nn;
  parent.assign(nn, EMPTY);
  inner.assign(nn, NEVER);
  inner[0] = 0;
  for (size_t i = 0; i < nn; ++i) {  // children follow their parents
    if (inner[i] == NEVER) continue;
    for (int c = 0; c < 4; ++c) {
      const uint32_t id = nodes[i * TOP_WORDS + 24 + c];
      if (id == EMPTY || (id & LEAF)) continue;
      if (id >= nn) {
        need = std::max<size_t>(need, (size_t)id + 1);
        continue;
      }
      if (id <= i || inner[id] != NEVER) continue;  // words that are no tree from node 0: the child's box as it stands
      parent[id] = (uint32_t)i, inner[id] = 0, ++inner[i];
    }
  }
  return need;
}

}  // namespace

extern "C" rt_status rt_scene_move_instances(rt_ctx* ctx, rt_scene* scene, const rt_instance* instances, uint32_t n,
                                             const float* mesh_boxes, uint32_t n_meshes, void* stream) {
  if (!ctx || !scene || (n && !instances) || (n_meshes && !mesh_boxes)) return fail(ctx, RT_ERR_INVALID_ARG, "null argument");
  if (scene->layout > 1) return fail(ctx, RT_ERR_UNSUPPORTED, "instances move in the BVH4 layouts");
  const uint32_t layout = scene->layout;
  std::lock_guard<std::mutex> lock(ctx->mu);
  RT_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  RT_CUDA(ctx, cudaStreamIsCapturing(s, &capture));
  if (capture != cudaStreamCaptureStatusNone) return fail(ctx, RT_ERR_CUDA, "a move cannot be captured: it reads host arrays");
  const uint32_t* head = scene->head;
  const uint32_t count = head[0];
  if (n != count || (layout == 0 && head[4] > count))  // GI word 4: a see-through tail
    return fail(ctx, RT_ERR_INVALID_ARG, "moved instances must be the scene's %u instances, in record order", count);
  for (uint32_t i = 0; i < n; ++i) {
    const rt_instance& s = instances[i];
    if (s.mesh >= n_meshes) return fail(ctx, RT_ERR_INVALID_ARG, "instance %u: mesh %u of %u", i, s.mesh, n_meshes);
    if (rtb::is_singular(s.model, s.rows)) return fail(ctx, RT_ERR_LAYOUT, "instance %u: singular placement", i);
  }
  if (n == 0) return RT_OK;
  // All that can be refused or fail comes before the first launch, and the refit count is written where
  // the refit or the rebuild is: a call that fails in between leaves the count as it was.
  const size_t base = layout == 0 ? head[1] : (head[1] & ~3u);
  const bool top = head[1] != 0 && count >= 2, rebuild = top && head[3] >= rtb::TLAS_REFITS;
  const size_t span = top ? rtb::tlas_reserve(count) : 0;
  if (top && base + span > scene->n_words) return fail(ctx, RT_ERR_LAYOUT, "top level exceeds the scene's words");
  if (layout == 1 && (size_t)head[4] + 8 > scene->n_words) return fail(ctx, RT_ERR_LAYOUT, "scene bounds exceed the words");
  const size_t need = sizeof(rt_instance) * n + 24 * (size_t)n_meshes;
  if (need > scene->move_bytes) {
    RT_CUDA(ctx, wait_changes(scene));
    RT_CUDA(ctx, cudaFree(scene->d_move));
    scene->d_move = nullptr;
    scene->device_bytes -= scene->move_bytes;
    ctx->scene_bytes -= scene->move_bytes;
    scene->move_bytes = 0;
    if (device_alloc(ctx, &scene->d_move, need, true) != cudaSuccess) {
      cudaGetLastError();
      return fail(ctx, RT_ERR_OOM, "move staging (%zu bytes)", need);
    }
    scene->move_bytes = need;
    scene->device_bytes += need;
    ctx->scene_bytes += need;
  }
  // the top level's links, per node its parent, a counter, and (bytes) its inner children; the tree's
  // topology is read once (a rebuild keeps its own)
  std::vector<uint32_t> nodes, up;
  std::vector<uint8_t> kids;
  if (top && (scene->top_nodes == 0 || rebuild)) {
    size_t cap = span / TOP_WORDS;  // a rebuild's most
    if (!rebuild) {
      RT_CUDA(ctx, wait_changes(scene));
      for (size_t seen = 0; seen < cap;) {
        seen = cap;
        nodes.resize(cap * TOP_WORDS);
        RT_CUDA(ctx, cudaMemcpy(nodes.data(), scene->d_words + base, 4 * nodes.size(), cudaMemcpyDeviceToHost));
        cap = std::min(top_links(nodes, up, kids), (scene->n_words - base) / TOP_WORDS);
      }
    }
    if (cap > scene->top_cap) {
      RT_CUDA(ctx, wait_changes(scene));
      RT_CUDA(ctx, cudaFree(scene->d_top_tree));
      scene->d_top_tree = nullptr, scene->top_cap = 0, scene->top_nodes = 0;
      if (device_alloc(ctx, &scene->d_top_tree, 9 * cap, true) != cudaSuccess) {
        cudaGetLastError();
        scene->d_top_tree = nullptr;
        return fail(ctx, RT_ERR_OOM, "top-level links");
      }
      scene->top_cap = cap;
    }
  }
  uint32_t *parent = scene->d_top_tree, *done = parent + scene->top_cap;
  uint8_t* inner = reinterpret_cast<uint8_t*>(done + scene->top_cap);
  if (!up.empty()) {
    RT_CUDA(ctx, cudaMemcpy(parent, up.data(), 4 * up.size(), cudaMemcpyHostToDevice));
    RT_CUDA(ctx, cudaMemcpy(inner, kids.data(), kids.size(), cudaMemcpyHostToDevice));
    scene->top_nodes = (uint32_t)up.size();
  }
  rt_instance* d_moved = static_cast<rt_instance*>(scene->d_move);
  float* d_boxes = reinterpret_cast<float*>(d_moved + n);
  Change change(scene, s);
  RT_CUDA(ctx, change.start());
  // one copy, from memory of the scene's own, whatever memory the caller's arrays are in; the last
  // call's copy has to have read it
  RT_CUDA(ctx, wait_changes(scene));
  scene->move_stage.resize(need);
  std::memcpy(scene->move_stage.data(), instances, sizeof(rt_instance) * n);
  if (n_meshes) std::memcpy(scene->move_stage.data() + sizeof(rt_instance) * n, mesh_boxes, 24 * (size_t)n_meshes);
  scene->w8_top_valid = false;  // the instances move: the packed top level until re-prepared
  RT_CUDA(ctx, cudaMemcpyAsync(d_moved, scene->move_stage.data(), need, cudaMemcpyHostToDevice, s));
  k_move_records<<<(n + 127) / 128, 128, 0, s>>>(scene->d_words, layout, d_moved, n, d_boxes);
  RT_CUDA(ctx, cudaGetLastError());
  if (rebuild) {
    // Rebuilt on the device from the records' new boxes (instance_bvh::place for a moved set).
    const size_t header = layout == 0 ? 16 : 8, stride = layout == 0 ? 32 : 24;
    uint32_t n_nodes = 0;
    scene->top_nodes = 0;
    const rt_status st = tlas_build_device(ctx, scene->d_words + header + 12, stride, n, true, scene->d_words + base, span,
                                           &n_nodes, s);
    if (st != RT_OK) return st;
    k_top_links<<<(n_nodes + 127) / 128, 128, 0, s>>>(scene->d_words, base, n_nodes, parent, inner);
    RT_CUDA(ctx, cudaGetLastError());
    scene->head[3] = 0;
    scene->top_nodes = n_nodes;
  } else if (top) {
    RT_CUDA(ctx, cudaMemsetAsync(done, 0, 4 * (size_t)scene->top_nodes, s));
    k_refit_top<<<(4 * scene->top_nodes + TOP_BLOCK - 1) / TOP_BLOCK, TOP_BLOCK, 0, s>>>(
        scene->d_words, layout, base, scene->top_nodes, parent, inner, done, scene->head[3] + 1);
    RT_CUDA(ctx, cudaGetLastError());
    scene->head[3] += 1;
  }
  if (layout == 1) {
    k_scene_bounds<<<1, BOUNDS_THREADS, 0, s>>>(scene->d_words, n);
    RT_CUDA(ctx, cudaGetLastError());
  }
  return RT_OK;
}
