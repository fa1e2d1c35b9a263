// FAST traversal kernels: the PLAIN per-ray arithmetic and visit order, rescheduled.
//
// Each ray performs exactly the operations of rs_trace / gi_traverse in the same order (so its
// hit is bit-identical), but the loop is flattened into a per-lane state machine -- one top-level
// node, instance entry, BLAS node or leaf a step -- inside persistent warps that refill lanes with
// new rays as rays end (warp-aggregated atomics on a global ray counter).
//
// What bounds them: instruction issue. Lanes of one warp wait for different kinds of step, and a
// warp that runs every kind each time around executes each for a fourth of its lanes (6.7 of 32
// active on 1.05M gather rays over 400 instances, 59 % of issue slots taken, 6.3 G instructions).
// So the warp votes and runs the one step that most lanes wait for, the others keep theirs
// (vote_phase): 11.9 lanes active, 4.3 G instructions. Running every step with at least 6, 8 or 12
// lanes waiting as well was slower (6.78, 6.35 and 6.23 against 6.08 ms there), and so were weights
// by a step's length. Each is resident 7 times an SM (72 registers): 4, 5, 6 and 8 blocks gave 6.65,
// 6.63, 6.10 and 6.12 against 6.09 ms; the closest hit therefore keeps no more than t, u, v and where
// its triangle is, and the record is made when the ray ends. Together, before and after (us):
//   gather of 16,384 cells over 400 instances, closest   9,530 -> 6,160
//   16,384 cells x 40 lights, 250k triangles, any hit      508 ->   438
//   1M GI rays, 250k triangles, GI / reflection          1,876 / 1,455 -> 1,320 / 1,000
//   1M camera rays, the same scene                         989 /   765 ->   765 /   600
#pragma once
#include "plain.cuh"

namespace rtk {

constexpr int FAST_MIN_BLOCKS = 7;  // of 128 threads an SM (72 registers)

// Persistent-kernel ray distribution: every lane that needs a ray takes the next index of the
// launch; one atomic per warp per refill round.
struct RayQueue {
  unsigned int* next;  // global counter, zeroed before the launch
  uint32_t n;
  uint32_t refill;     // idle lanes a warp waits for before taking more rays (1-width)
  uint32_t width;      // lanes of a warp that take rays (1-32): fewer than 32 where n rays do not fill the GPU
};

// Called by all 32 lanes together. `drained` (warp-uniform) stops the requests once the
// counter has passed the end, so finished warps add no atomic traffic.
RT_DEV uint32_t take_ray(const RayQueue& q, bool need, bool& drained) {
  const unsigned idle = __ballot_sync(0xffffffffu, need && (threadIdx.x & 31) < q.width);
  const unsigned want = (!drained && (uint32_t)__popc(idle) >= q.refill) ? idle : 0u;
  if (!want) return EMPTY;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(want) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(q.next, (unsigned)__popc(want));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (base + (uint32_t)__popc(want) >= q.n) drained = true;
  const uint32_t idx = base + __popc(want & ((1u << lane) - 1u));
  return ((want >> lane & 1u) && idx < q.n) ? idx : EMPTY;
}

// ---------------------------------------------------------------- the walk's schedule

// Byte c of `word` as a float, exactly: as_float(0x4B000000 | q) - 2^23.
RT_DEV float byte_f(uint32_t word, uint32_t c) {
  return __fsub_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u | c)), 8388608.0f);
}

// slab_near of a BVH4-Q8 node's four children, planes decoded as base + q * step with each product
// and sum rounded on its own (see P2: the products are taken one by one), the sums and the rest two
// children to an instruction. 1M GI rays, reflection: 1,000 us against 1,050 one child at a time.
RT_DEV void child_slabs(F3 base, F3 step, uint32_t lx, uint32_t ly, uint32_t lz, uint32_t hx, uint32_t hy, uint32_t hz, F3 o,
                        F3 inv, float tmin, float tmax, float (&dist)[4]) {
#pragma unroll
  for (uint32_t c = 0; c < 4; c += 2) {
    auto plane = [&](uint32_t word, float b, float s, float at, float iv) {
      return mul2(add2(add2(pack2(mul(byte_f(word, c), s), mul(byte_f(word, c + 1), s)), both(b)), both(-at)), both(iv));
    };
    const P2 ax = plane(lx, base.x, step.x, o.x, inv.x), bx = plane(hx, base.x, step.x, o.x, inv.x);
    const P2 ay = plane(ly, base.y, step.y, o.y, inv.y), by = plane(hy, base.y, step.y, o.y, inv.y);
    const P2 az = plane(lz, base.z, step.z, o.z, inv.z), bz = plane(hz, base.z, step.z, o.z, inv.z);
    auto entry = [&](float x0, float x1, float y0, float y1, float z0, float z1) {
      const float near = fmaxf(fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1)), tmin);
      const float far = fminf(fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1)), tmax);
      return near <= far ? near : BIG;
    };
    dist[c] = entry(first(ax), first(bx), first(ay), first(by), first(az), first(bz));
    dist[c + 1] = entry(second(ax), second(bx), second(ay), second(by), second(az), second(bz));
  }
}

// ---------------------------------------------------------------- reflection layout

template <int AM>
struct RsLane {
  Ray ray;
  F3 world_inv;
  RsBest best;
  uint32_t ray_id;
  uint32_t entry;  // batch entry (many-batch launches)
  bool any;        // any-hit ray (AM 2)
  uint32_t phase;
  uint32_t top_at;  // items on the top level's stack, or the next instance of a flat list
  uint32_t inst, slot;
  F3 o, d, inv;
  uint32_t nodes, tris;
  uint32_t cur;  // what the next step works on: top-level node, instance, BLAS node or leaf
  uint32_t sp;
};

// The next item of the top level (or of the flat instance list).
template <class Lane>
RT_DEV void next_top(Lane& L, const uint32_t* top_stack, bool flat, uint32_t instances) {
  if (flat) {
    if (L.top_at >= instances) {
      L.phase = PH_DONE;
    } else {
      L.cur = L.top_at++;
      L.phase = PH_ENTER;
    }
    return;
  }
  if (L.top_at == 0) {
    L.phase = PH_DONE;
    return;
  }
  const uint32_t item = top_stack[--L.top_at];
  L.cur = item & ~LEAF;
  L.phase = (item & LEAF) ? PH_ENTER : PH_TOP;
}

template <class Lane>
RT_DEV void set_child(Lane& L, uint32_t child) {
  L.cur = child;
  L.phase = (child & LEAF) ? PH_LEAF : PH_NODE;
}

template <int AM, class Src>
RT_DEV void rs_finish(const RsLane<AM>& L, const Src& src) {
  if (any_of<AM>(L)) {
    put_flag(src, L.entry, L.ray_id, L.ray, L.best.rec[0] != 0);
    return;
  }
  uint32_t* o = reinterpret_cast<uint32_t*>(out_of(src, L.entry)) + 5 * (size_t)L.ray_id;
  o[0] = __float_as_uint(L.best.t), o[1] = L.best.rec[0], o[2] = L.best.rec[1], o[3] = L.best.rec[2];
  o[4] = L.best.rec[3];
}

// rs_instance's entry (reflections_software_bvh4.wgsl:50-67): true when the lane now walks the
// instance's BLAS.
template <int AM>
RT_DEV bool rs_enter(const uint32_t* __restrict__ w, RsLane<AM>& L, uint32_t i) {
  const size_t R = 8 + (size_t)i * 24;
  const uint4 tail = ld4(w, R + 20);
  if (any_of<AM>(L) && tail.z != 0) return false;
  const uint4 b0 = ld4(w, R + 12), b1 = ld4(w, R + 16);
  const float bound = rs_limit(L.best, i);
  const F3 lo = {__uint_as_float(b0.x), __uint_as_float(b0.y), __uint_as_float(b0.z)};
  const F3 hi = {__uint_as_float(b0.w), __uint_as_float(b1.x), __uint_as_float(b1.y)};
  if (slab_near(L.ray.o, L.world_inv, lo, hi, L.ray.tmin, bound) > bound) return false;
  to_object(ld4(w, R), ld4(w, R + 4), ld4(w, R + 8), L.ray, L.o, L.d);
  L.inv = safe_inverse(L.d);
  L.nodes = b1.z & ~3u;
  L.tris = b1.w & ~3u;
  L.inst = i;
  L.slot = tail.y;
  L.sp = 0;
  set_child(L, tail.x);
  return true;
}

// One leaf (reflections_software_bvh4.wgsl:72-95). True when an any-hit ray is blocked.
template <int AM>
RT_DEV bool rs_leaf(const uint32_t* __restrict__ w, RsLane<AM>& L, uint32_t child) {
  const uint32_t start = (child & ~LEAF) >> 4, count = child & 15u;
  const F3 o = L.o, d = L.d;
  for (uint32_t k = 0; k < count; ++k) {
    const size_t X = L.tris + (size_t)(start + k) * 12;
    const uint4 w0 = ld4(w, X), w1 = ld4(w, X + 4), w2 = ld4(w, X + 8);
    const F3 a = {__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z)};
    const F3 e1 = {__uint_as_float(w0.w), __uint_as_float(w1.x), __uint_as_float(w1.y)};
    const F3 e2 = {__uint_as_float(w1.z), __uint_as_float(w1.w), __uint_as_float(w2.x)};
    const F3 p = cross3(d, e2);
    const float det = dot3(e1, p);
    if (fabsf(det) < 1e-30f) continue;
    const float inv_det = __frcp_rn(det);
    const F3 s = sub3(o, a);
    const float u = mul(dot3(s, p), inv_det);
    if (u < -RS_EDGE || u > 1.0f + RS_EDGE) continue;
    const F3 q = cross3(s, e1);
    const float v = mul(dot3(d, q), inv_det);
    if (v < -RS_EDGE || add(u, v) > 1.0f + RS_EDGE) continue;
    const float t = mul(dot3(e2, q), inv_det);
    const bool tied = L.best.rec[0] != 0 && t == L.best.t &&
                      (L.inst < L.best.inst || (L.inst == L.best.inst && w2.y < L.best.rec[1]));
    if (t > L.ray.tmin && (t < L.best.t || tied)) {
      L.best.t = t;
      L.best.rec[0] = L.slot + 1, L.best.rec[1] = w2.y, L.best.rec[2] = __float_as_uint(u);
      L.best.rec[3] = __float_as_uint(v);
      L.best.inst = L.inst;
      if (any_of<AM>(L)) return true;
    }
  }
  return false;
}

// One BLAS node (reflections_software_bvh4.wgsl:99-125): children sorted, the nearest returned
// (EMPTY: none survives), the rest pushed far to near.
template <int AM>
RT_DEV uint32_t rs_node(const uint32_t* __restrict__ w, RsLane<AM>& L, uint32_t child, uint32_t* stack, DevStatus* st) {
  const size_t N = L.nodes + (size_t)child * 16;
  const uint4 n0 = ld4(w, N), n1 = ld4(w, N + 4), n2 = ld4(w, N + 8), n3 = ld4(w, N + 12);
  const float lim = rs_limit(L.best, L.inst);
  uint32_t ids[4] = {n1.z, n1.w, n2.x, n2.y};
  float dist[4];
  child_slabs({__uint_as_float(n0.x), __uint_as_float(n0.y), __uint_as_float(n0.z)},
              {__uint_as_float(n0.w), __uint_as_float(n1.x), __uint_as_float(n1.y)}, n2.z, n2.w, n3.x, n3.y, n3.z, n3.w, L.o,
              L.inv, L.ray.tmin, lim, dist);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (ids[c] == EMPTY) dist[c] = BIG;
#define RT_SW(a, b)                                      \
  if (dist[b] < dist[a]) {                               \
    float x = dist[a]; dist[a] = dist[b]; dist[b] = x;   \
    uint32_t y = ids[a]; ids[a] = ids[b]; ids[b] = y;    \
  }
  RT_SW(0, 1) RT_SW(2, 3) RT_SW(0, 2) RT_SW(1, 3) RT_SW(1, 2)
#undef RT_SW
#pragma unroll
  for (int c = 3; c >= 1; --c) {
    if (dist[c] <= lim && ids[c] != EMPTY) {
      if (L.sp < STACK) stack[L.sp++] = ids[c];
      else atomicAdd(&st->stack_drops, 1ull);
    }
  }
  return dist[0] <= lim ? ids[0] : EMPTY;
}

template <int AM, int BLOCK, class Src>
__global__ void __launch_bounds__(BLOCK, FAST_MIN_BLOCKS)
    k_rs_fast(const uint32_t* __restrict__ w, const Src src, RayQueue queue, DevStatus* st) {
  uint32_t stack[STACK];
  uint32_t top_stack[STACK];
  RsLane<AM> L;
  L.phase = PH_IDLE;
  const uint4 head = ld4(w, 0);
  const size_t bounds = ld(w, 4) & ~3u;
  const size_t top = head.y & ~3u;
  bool drained = false;
  for (;;) {
    // Every lane reaches the votes below once per iteration (no exit above them); the warp leaves
    // only when no lane holds a ray and the queue is drained.
    __syncwarp();
    const uint32_t id = take_ray(queue, L.phase == PH_IDLE || L.phase == PH_DONE, drained);
    if (id != EMPTY) {
      if (L.phase == PH_DONE) rs_finish<AM>(L, src);
      L.ray = fetch(src, id, L);
      L.world_inv = safe_inverse(L.ray.d);
      L.best.t = L.ray.tmax, L.best.rec[0] = L.best.rec[1] = L.best.rec[2] = L.best.rec[3] = 0, L.best.inst = EMPTY;
      // rs_trace prologue (reflections_software_bvh4.wgsl:141-155)
      bool live = head.x != 0;
      if (live) {
        const F3 lo = ld3(w, bounds), hi = ld3(w, bounds + 4);
        const F3 o = L.ray.o, wi = L.world_inv;
        const float ax = mul(sub(lo.x, o.x), wi.x), ay = mul(sub(lo.y, o.y), wi.y), az = mul(sub(lo.z, o.z), wi.z);
        const float bx = mul(sub(hi.x, o.x), wi.x), by = mul(sub(hi.y, o.y), wi.y), bz = mul(sub(hi.z, o.z), wi.z);
        const float near = fmaxf(fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz)), L.ray.tmin);
        const float far = fminf(fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz)), L.ray.tmax);
        live = !(near > far);
        if (live) L.best.t = fminf(L.ray.tmax, __uint_as_float(__float_as_uint(far) + 2u));
      }
      L.phase = PH_DONE;  // misses the scene box
      if (live) {
        L.top_at = head.y == 0 ? 0 : 1;
        top_stack[0] = head.z;
        next_top(L, top_stack, head.y == 0, head.x);
      }
    }
    const uint32_t run = vote_phase(L.phase);
    if (run == PH_IDLE) {
      if (drained) break;
      continue;
    }
    if (L.phase != run) continue;
    if (run == PH_NODE) {
      const uint32_t c = rs_node<AM>(w, L, L.cur, stack, st);
      if (c != EMPTY) set_child(L, c);
      else if (L.sp) set_child(L, stack[--L.sp]);
      else next_top(L, top_stack, head.y == 0, head.x);
    } else if (run == PH_LEAF) {
      if (rs_leaf<AM>(w, L, L.cur)) L.phase = PH_DONE;
      else if (L.sp) set_child(L, stack[--L.sp]);
      else next_top(L, top_stack, head.y == 0, head.x);
    } else if (run == PH_ENTER) {
      if (!rs_enter<AM>(w, L, L.cur)) next_top(L, top_stack, head.y == 0, head.x);
    } else {
      const float bound = L.best.rec[0] != 0 ? next_up(L.best.t) : L.best.t;
      top_step(w, top + (size_t)L.cur * 32, L.ray, L.world_inv, bound, top_stack, L.top_at, st);
      next_top(L, top_stack, false, 0);
    }
  }
  if (L.phase == PH_DONE) rs_finish<AM>(L, src);
}

// ---------------------------------------------------------------- GI layout

// The closest hit so far: the record's identity words and normal are made once, when the ray ends.
struct GiNear {
  float t, u, v;
  uint32_t inst;  // EMPTY: none
  uint32_t at;    // word of the triangle's three indices
};
RT_DEV float gi_limit(const GiNear& b, uint32_t i) { return (b.inst != EMPTY && i < b.inst) ? next_up(b.t) : b.t; }

template <int AM>
struct GiLane {
  Ray ray;
  F3 world_inv;
  GiNear best;
  uint32_t ray_id;
  uint32_t entry;
  bool any;
  uint32_t phase;
  uint32_t top_at;
  uint32_t inst;
  F3 o, d, inv;
  uint32_t nodes, leaves, positions, indices;
  uint32_t cur, sp;
};

// The record of an ended ray (gi_rays_software.wgsl:141-169): a hit's primitive or position
// indices, and the world normal of its source winding.
template <int AM, class Src>
RT_DEV void gi_finish(const uint32_t* __restrict__ w, const GiLane<AM>& L, const Src& src) {
  const GiNear& b = L.best;
  if (any_of<AM>(L)) {
    put_flag(src, L.entry, L.ray_id, L.ray, b.inst != EMPTY);
    return;
  }
  uint32_t* o = reinterpret_cast<uint32_t*>(out_of(src, L.entry)) + 10 * (size_t)L.ray_id;
  uint32_t tri[3] = {0, 0, 0};
  F3 n = {0.0f, 0.0f, 0.0f};
  if (b.inst != EMPTY) {
    const size_t r = 16 + (size_t)b.inst * 32;
    const uint32_t positions = ld(w, r + 20), indices = ld(w, r + 21), prim_base = ld(w, r + 28);
    tri[0] = ld(w, b.at), tri[1] = ld(w, (size_t)b.at + 1), tri[2] = ld(w, (size_t)b.at + 2);
    const F3 a = ld3(w, positions + (size_t)tri[0] * 3), bb = ld3(w, positions + (size_t)tri[1] * 3),
             c = ld3(w, positions + (size_t)tri[2] * 3);
    const F3 cr = cross3(sub3(bb, a), sub3(c, a));
    const uint4 q0 = ld4(w, r), q1 = ld4(w, r + 4), q2 = ld4(w, r + 8);
    n = unit_normal({add(add(mul(__uint_as_float(q0.x), cr.x), mul(__uint_as_float(q1.x), cr.y)), mul(__uint_as_float(q2.x), cr.z)),
                     add(add(mul(__uint_as_float(q0.y), cr.x), mul(__uint_as_float(q1.y), cr.y)), mul(__uint_as_float(q2.y), cr.z)),
                     add(add(mul(__uint_as_float(q0.z), cr.x), mul(__uint_as_float(q1.z), cr.y)), mul(__uint_as_float(q2.z), cr.z))});
    if (prim_base != 0) tri[0] = ld(w, prim_base + (b.at - indices) / 3), tri[1] = 0, tri[2] = 0;
  }
  o[0] = __float_as_uint(b.t), o[1] = b.inst, o[2] = tri[0], o[3] = tri[1], o[4] = tri[2];
  o[5] = __float_as_uint(b.u), o[6] = __float_as_uint(b.v);
  o[7] = __float_as_uint(n.x), o[8] = __float_as_uint(n.y), o[9] = __float_as_uint(n.z);
}

// gi_instance's entry (gi_rays_software.wgsl:100-113): true when the lane now walks the
// instance's BLAS.
template <int AM>
RT_DEV bool gi_enter(const uint32_t* __restrict__ w, GiLane<AM>& L, uint32_t i) {
  const size_t r = 16 + (size_t)i * 32;  // records start on 16 bytes
  if (any_of<AM>(L) && (ld(w, r + 27) & 1u) != 0) return false;
  const uint4 b0 = ld4(w, r + 12), b1 = ld4(w, r + 16);
  const float lim = gi_limit(L.best, i);
  const F3 lo = {__uint_as_float(b0.x), __uint_as_float(b0.y), __uint_as_float(b0.z)};
  const F3 hi = {__uint_as_float(b0.w), __uint_as_float(b1.x), __uint_as_float(b1.y)};
  if (!(slab_near(L.ray.o, L.world_inv, lo, hi, L.ray.tmin, lim) <= lim)) return false;
  const uint4 b2 = ld4(w, r + 20);
  to_object(ld4(w, r), ld4(w, r + 4), ld4(w, r + 8), L.ray, L.o, L.d);
  L.inv = safe_inverse(L.d);
  L.nodes = b1.z, L.leaves = b1.w, L.positions = b2.x, L.indices = b2.y;
  L.inst = i;
  L.sp = 0;
  set_child(L, b2.z);
  return true;
}

// One GI leaf (gi_rays_software.wgsl:117-169). True when an any-hit ray is blocked.
template <int AM>
RT_DEV bool gi_leaf(const uint32_t* __restrict__ w, GiLane<AM>& L, uint32_t child) {
  const size_t l = L.leaves + (size_t)(child & ~LEAF) * 2;
  const uint32_t first = ld(w, l), count = ld(w, l + 1);
  const uint32_t i = L.inst;
  for (uint32_t k = 0; k < count; k += 6) {
    const uint32_t x = L.indices + first + k;
    const bool two = k + 3 < count;
    const uint32_t y = two ? x + 3 : x;
    const uint32_t ia = ld(w, x), ib = ld(w, x + 1), ic = ld(w, x + 2);
    const uint32_t ja = ld(w, y), jb = ld(w, y + 1), jc = ld(w, y + 2);
    const F3 a = ld3(w, L.positions + (size_t)ia * 3), b = ld3(w, L.positions + (size_t)ib * 3),
             c = ld3(w, L.positions + (size_t)ic * 3);
    const F3 a2 = ld3(w, L.positions + (size_t)ja * 3), b2 = ld3(w, L.positions + (size_t)jb * 3),
             c2 = ld3(w, L.positions + (size_t)jc * 3);
    float t, u, v;
    if (gi_triangle(L.o, L.d, a, b, c, L.ray.tmin, gi_limit(L.best, i), t, u, v)) {
      L.best = GiNear{t, u, v, i, x};
      if (any_of<AM>(L)) return true;
    }
    if (two && gi_triangle(L.o, L.d, a2, b2, c2, L.ray.tmin, gi_limit(L.best, i), t, u, v)) {
      L.best = GiNear{t, u, v, i, y};
      if (any_of<AM>(L)) return true;
    }
  }
  return false;
}

// One GI BLAS node (gi_rays_software.wgsl:171-204): every surviving child pushed far to near; the
// nearest of them is returned instead (it would be popped next), EMPTY when none survives.
template <int AM>
RT_DEV uint32_t gi_node(const uint32_t* __restrict__ w, GiLane<AM>& L, uint32_t child, uint32_t* stack, DevStatus* st) {
  const size_t n = L.nodes + (size_t)child * 16;
  uint4 nn[4];
  ld16(w, n, nn);
  const uint4 &n0 = nn[0], &n1 = nn[1], &n2 = nn[2], &n3 = nn[3];
  uint32_t c[4] = {n1.z, n1.w, n2.x, n2.y};
  const float lim = gi_limit(L.best, L.inst);
  float dist[4];
  child_slabs({__uint_as_float(n0.x), __uint_as_float(n0.y), __uint_as_float(n0.z)},
              {__uint_as_float(n0.w), __uint_as_float(n1.x), __uint_as_float(n1.y)}, n2.z, n2.w, n3.x, n3.y, n3.z, n3.w, L.o,
              L.inv, L.ray.tmin, lim, dist);
  uint32_t tb[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) tb[s] = __float_as_uint(c[s] == EMPTY ? BIG : dist[s]);
#define RT_SW(a, b)                          \
  if (tb[a] < tb[b]) {                       \
    uint32_t x = tb[a]; tb[a] = tb[b]; tb[b] = x; \
    x = c[a]; c[a] = c[b]; c[b] = x;         \
  }
  RT_SW(0, 1) RT_SW(2, 3) RT_SW(0, 2) RT_SW(1, 3) RT_SW(1, 2)
#undef RT_SW
  uint32_t next = EMPTY;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    if (__uint_as_float(tb[s]) <= lim && c[s] != EMPTY) {
      if (next != EMPTY) stack[L.sp++] = next;
      next = c[s];
      if (L.sp >= STACK) next = EMPTY, atomicAdd(&st->stack_drops, 1ull);
    }
  }
  return next;
}

template <int AM, int BLOCK, class Src>
__global__ void __launch_bounds__(BLOCK, FAST_MIN_BLOCKS)
    k_gi_fast(const uint32_t* __restrict__ w, const Src src, RayQueue queue, DevStatus* st) {
  uint32_t stack[STACK];
  uint32_t top_stack[STACK];
  GiLane<AM> L;
  L.phase = PH_IDLE;
  const uint32_t instances = ld(w, 0), top = ld(w, 1), root = ld(w, 2);
  bool drained = false;
  for (;;) {
    __syncwarp();
    const uint32_t id = take_ray(queue, L.phase == PH_IDLE || L.phase == PH_DONE, drained);
    if (id != EMPTY) {
      if (L.phase == PH_DONE) gi_finish<AM>(w, L, src);
      L.ray = fetch(src, id, L);
      L.world_inv = safe_inverse(L.ray.d);
      L.best = GiNear{L.ray.tmax, 0.0f, 0.0f, EMPTY, 0u};
      L.top_at = top == 0 ? 0 : 1;
      top_stack[0] = root;
      next_top(L, top_stack, top == 0, instances);
    }
    const uint32_t run = vote_phase(L.phase);
    if (run == PH_IDLE) {
      if (drained) break;
      continue;
    }
    if (L.phase != run) continue;
    if (run == PH_NODE) {
      const uint32_t c = gi_node<AM>(w, L, L.cur, stack, st);
      if (c != EMPTY) set_child(L, c);
      else if (L.sp) set_child(L, stack[--L.sp]);
      else next_top(L, top_stack, top == 0, instances);
    } else if (run == PH_LEAF) {
      if (gi_leaf<AM>(w, L, L.cur)) L.phase = PH_DONE;
      else if (L.sp) set_child(L, stack[--L.sp]);
      else next_top(L, top_stack, top == 0, instances);
    } else if (run == PH_ENTER) {
      if (!gi_enter<AM>(w, L, L.cur)) next_top(L, top_stack, top == 0, instances);
    } else {
      const float bound = L.best.inst != EMPTY ? next_up(L.best.t) : L.best.t;
      top_step(w, top + (size_t)L.cur * 32, L.ray, L.world_inv, bound, top_stack, L.top_at, st);
      next_top(L, top_stack, false, 0);
    }
  }
  if (L.phase == PH_DONE) gi_finish<AM>(w, L, src);
}

}  // namespace rtk
