// The BVH4-Q8 node quantiser on the device, shared by the GPU refit and the GPU build: child boxes
// formed as the host builder forms them (a leaf's vertices in index order; an inner child's
// decoded planes, unfused and fused, over its children in slot order) and quantize_node's exact
// arithmetic (near_field.rs:402-430, 481-525), every step an explicit round-to-nearest operation,
// so the node words equal the host's bit for bit.
#pragma once
#include <cuda_runtime.h>

#include <cfloat>
#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace rtq {

using rtk::EMPTY;
using rtk::LEAF;

struct Box {
  float lo[3], hi[3];
};

// f32::min / f32::max as the host builders write them (the first operand wins a tie).
__device__ __forceinline__ float lo_of(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float hi_of(float a, float b) { return b > a ? b : a; }
__device__ __forceinline__ void grow(Box& b, float x, float y, float z) {
  b.lo[0] = lo_of(b.lo[0], x), b.lo[1] = lo_of(b.lo[1], y), b.lo[2] = lo_of(b.lo[2], z);
  b.hi[0] = hi_of(b.hi[0], x), b.hi[1] = hi_of(b.hi[1], y), b.hi[2] = hi_of(b.hi[2], z);
}
__device__ __forceinline__ Box empty_box() { return Box{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}}; }
// A decoded plane, unfused (origin + step * q) or fused (fma).
__device__ __forceinline__ float plane(float o, float s, uint32_t q, bool fused) {
  return fused ? __fmaf_rn(s, (float)q, o) : __fadd_rn(o, __fmul_rn(s, (float)q));
}
__device__ __forceinline__ uint32_t to_u8(float f) {  // `f.clamp(0.0, 255.0) as u8`
  if (!(f > 0.0f)) return 0;
  if (f >= 255.0f) return 255;
  return (uint32_t)f;
}

struct View {
  uint32_t* w;
  uint32_t layout;
  size_t nodes, leaves, positions, indices;  // GI word offsets of the BLAS
  size_t tris;                               // reflection: its triangles
  const float* pos;                          // reflection: the new positions
  const uint32_t* src;                       // reflection: the source triangle list
};

__device__ __forceinline__ void grow_vertex(const View& v, Box& b, uint32_t vi, bool from_words) {
  if (from_words) {
    const uint32_t* p = v.w + v.positions + 3 * (size_t)vi;
    grow(b, __uint_as_float(p[0]), __uint_as_float(p[1]), __uint_as_float(p[2]));
  } else {
    const float* p = v.pos + 3 * (size_t)vi;
    grow(b, p[0], p[1], p[2]);
  }
}

// The box of one child, as the host refit forms it: a leaf's vertices in index order; an inner
// child's decoded planes, unfused and fused, over its children in slot order.
inline __device__ Box child_box(const View& v, uint32_t c) {
  Box b = empty_box();
  if (c & LEAF) {
    if (v.layout == 0) {
      const size_t l = v.leaves + 2 * (size_t)(c & ~LEAF);
      const uint32_t first = v.w[l], count = v.w[l + 1];
      for (uint32_t k = first; k < first + count; ++k) grow_vertex(v, b, v.w[v.indices + k], true);
    } else {
      const uint32_t first = (c & ~LEAF) >> 4, count = c & 15u;
      for (uint32_t t = first; t < first + count; ++t) {
        const uint32_t prim = v.w[v.tris + 12 * (size_t)t + 9];
        for (int j = 0; j < 3; ++j) grow_vertex(v, b, v.src[3 * (size_t)prim + j], false);
      }
    }
    return b;
  }
  // another thread block may have written the child in this launch: past L1
  const uint32_t* p = v.w + v.nodes + 16 * (size_t)c;
  uint32_t n[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) n[k] = __ldcg(p + k);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    if (n[6 + t] == EMPTY) continue;
    for (int fused = 0; fused < 2; ++fused)
      for (int a = 0; a < 3; ++a) {
        const float o = __uint_as_float(n[a]), s = __uint_as_float(n[3 + a]);
        b.lo[a] = lo_of(b.lo[a], plane(o, s, (n[10 + a] >> (8 * t)) & 255u, fused));
        b.hi[a] = hi_of(b.hi[a], plane(o, s, (n[13 + a] >> (8 * t)) & 255u, fused));
      }
  }
  return b;
}

// One node by four lanes (`quad`: their mask, `c`: this lane's 0-3), a child each: the children's
// boxes, quantize_node's origin and step per axis, and each child's outward 8-bit planes. Minima and
// maxima prefer the earlier child of two equal values, as the host's sequential pass does.
inline __device__ void refit_node(const View& v, uint32_t node, unsigned quad, int c) {
  uint32_t* w = v.w + v.nodes + 16 * (size_t)node;
  const uint32_t id = w[6 + c];
  const bool here = id != EMPTY;
  const unsigned present = (__ballot_sync(quad, here) >> (__ffs(quad) - 1)) & 0xfu;
  const int n = __popc(present), k = __popc(present & ((1u << c) - 1u));  // k: the child's place among those present
  const Box box = here ? child_box(v, id) : empty_box();
  Box all = box;
  for (int step = 1; step < 4; step *= 2)
    for (int a = 0; a < 3; ++a) {
      const float lo = __shfl_xor_sync(quad, all.lo[a], step), hi = __shfl_xor_sync(quad, all.hi[a], step);
      all.lo[a] = (c & step) ? lo_of(lo, all.lo[a]) : lo_of(all.lo[a], lo);
      all.hi[a] = (c & step) ? hi_of(hi, all.hi[a]) : hi_of(all.hi[a], hi);
    }
  float mine = 0.0f;  // lanes 0-2: the step of one axis
  if (c < 3) {
    const float lo = c == 0 ? all.lo[0] : (c == 1 ? all.lo[1] : all.lo[2]), hi = c == 0 ? all.hi[0] : (c == 1 ? all.hi[1] : all.hi[2]);
    mine = hi_of(__fdiv_rn(__fsub_rn(hi, lo), 255.0f), hi_of(FLT_MIN, __fmul_rn(fabsf(lo), 1e-7f)));
    while (__fadd_rn(lo, __fmul_rn(mine, 255.0f)) < hi || __fmaf_rn(mine, 255.0f, lo) < hi)
      mine = __fmul_rn(mine, 1.0f + 1.0f / 1048576.0f);
  }
  const int first = __ffs(quad) - 1;
  uint32_t planes[6];  // lower x, y, z, upper x, y, z
  float steps[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float o = all.lo[a], s = __shfl_sync(quad, mine, first + a), x = box.lo[a], y = box.hi[a];
    steps[a] = s;
    uint32_t ql = 0, qh = 0;
    if (here) {
      ql = to_u8(floorf(__fdiv_rn(__fsub_rn(x, o), s)));
      while (ql > 0 && (plane(o, s, ql, false) > x || plane(o, s, ql, true) > x)) --ql;
      qh = to_u8(ceilf(__fdiv_rn(__fsub_rn(y, o), s)));
      while (qh < 255 && (plane(o, s, qh, false) < y || plane(o, s, qh, true) < y)) ++qh;
    }
    planes[a] = ql << (8 * k), planes[3 + a] = qh << (8 * k);
  }
  if (!here)  // places past the children present
    for (int a = 0; a < 6; ++a) planes[a] = 0;
  for (int step = 1; step < 4; step *= 2)
    for (int a = 0; a < 6; ++a) planes[a] |= __shfl_xor_sync(quad, planes[a], step);
  w[6 + (here ? k : n + c - k)] = here ? id : EMPTY;
  if (c < 3) {
    w[c] = __float_as_uint(c == 0 ? all.lo[0] : (c == 1 ? all.lo[1] : all.lo[2]));
    w[3 + c] = __float_as_uint(c == 0 ? steps[0] : (c == 1 ? steps[1] : steps[2]));
    w[10 + c] = c == 0 ? planes[0] : (c == 1 ? planes[1] : planes[2]);
    w[13 + c] = c == 0 ? planes[3] : (c == 1 ? planes[4] : planes[5]);
  }
}

constexpr uint8_t NEVER = 0xff;  // inner children of a node that the climb does not come to

// Nodes of one height above the leaves, four lanes each.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_refit_level(View v, const uint32_t* __restrict__ order, uint32_t count) {
  const uint32_t i = (blockIdx.x * BLOCK + threadIdx.x) / 4;
  if (i < count) refit_node(v, order[i], 0xfu << (threadIdx.x & 28), threadIdx.x & 3);
}

// Every node of a BLAS, children before parents, in one launch: four lanes start at each node without
// inner children (inner[node] == 0) and climb; of a node's inner children, the last one done takes
// the node (done[], zeroed before the launch). A launch per height had the upper heights wait on a
// few lone warps each: 250k triangles, 10 heights, 218 us against 60. Nothing waits.
constexpr int REFIT_BLOCK = 128;
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_refit_up(View v, uint32_t n, const uint32_t* __restrict__ parent,
                                                    const uint8_t* __restrict__ inner, uint32_t* __restrict__ done) {
  const uint32_t i = (blockIdx.x * BLOCK + threadIdx.x) / 4;
  if (i >= n || inner[i] != 0) return;
  const int c = threadIdx.x & 3;
  const unsigned quad = 0xfu << (threadIdx.x & 28);
  for (uint32_t node = i;;) {
    refit_node(v, node, quad, c);
    const uint32_t up = parent[node];
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
    node = up;
  }
}

}  // namespace rtq
