// PLAIN traversal kernels: one thread per ray, a 48-entry stack per thread, the WGSL loops
// statement for statement:
//   gi_traverse  -> shaders/gi_rays_software.wgsl:98-279 (opaque instances, BVH4 top level)
//   rs_trace     -> shaders/reflections_software_bvh4.wgsl:50-204
// Same arithmetic, same child order, same tie rules, so hits are bit-identical to the WGSL
// restatement. Two safety rules the WGSL leaves to robust buffer access: a child id EMPTY is
// never pushed, and a push onto a full stack is dropped and counted (DevStatus::stack_drops).
//
// The steps of a walk (instance entry, node, leaf) are shared with the FAST kernels (but for GI any hits in
// full warps: gi_blocked): records and nodes in 16-byte loads, slabs two children to an instruction,
// the GI hit record made when the ray ends. Closest hits, 1M camera rays over 120,000 cube triangles (GI)
// 234 -> 192 us, over 250k cluster triangles (reflection) 651 -> 553, 1M rays of uniform directions there
// 2,221 -> 1,803 (GI) and 1,688 -> 1,410.
#pragma once
#include "common.cuh"

namespace rtk {

// ---------------------------------------------------------------- shared steps

// The BVH4 top-level node step (gi_rays_software.wgsl:241-261, reflections_software_bvh4.wgsl
// :173-193): four slabs, the ascending five-exchange network, pushes far to near.
RT_DEV void top_step(const uint32_t* __restrict__ w, size_t n, const Ray& ray, F3 world_inv, float bound,
                     uint32_t* stack, uint32_t& sp, DevStatus* st) {
  float dist[4];
  uint32_t ids[4];
  // the node's seven 16-byte rows: lo x, lo y, lo z, hi x, hi y, hi z (four children each), ids
  const uint4 lx = ld4u(w, n), ly = ld4u(w, n + 4), lz = ld4u(w, n + 8);
  const uint4 hx = ld4u(w, n + 12), hy = ld4u(w, n + 16), hz = ld4u(w, n + 20), id4 = ld4u(w, n + 24);
  // two children to an instruction, each lane's difference and product rounded on its own
  auto plane = [](uint32_t a, uint32_t b, float o, float inv) {
    return mul2(add2(pack2(__uint_as_float(a), __uint_as_float(b)), both(-o)), both(inv));
  };
#pragma unroll
  for (int c = 0; c < 4; c += 2) {
    auto pair = [&](const uint4& q, float o, float inv) { return c == 0 ? plane(q.x, q.y, o, inv) : plane(q.z, q.w, o, inv); };
    const P2 ax = pair(lx, ray.o.x, world_inv.x), bx = pair(hx, ray.o.x, world_inv.x);
    const P2 ay = pair(ly, ray.o.y, world_inv.y), by = pair(hy, ray.o.y, world_inv.y);
    const P2 az = pair(lz, ray.o.z, world_inv.z), bz = pair(hz, ray.o.z, world_inv.z);
    auto entry = [&](float x0, float x1, float y0, float y1, float z0, float z1, uint32_t id) {
      const float near = fmaxf(fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1)), ray.tmin);
      const float far = fminf(fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1)), bound);
      return near <= far && id != EMPTY ? near : BIG;
    };
    ids[c] = c == 0 ? id4.x : id4.z, ids[c + 1] = c == 0 ? id4.y : id4.w;
    dist[c] = entry(first(ax), first(bx), first(ay), first(by), first(az), first(bz), ids[c]);
    dist[c + 1] = entry(second(ax), second(bx), second(ay), second(by), second(az), second(bz), ids[c + 1]);
  }
#define RT_SW(a, b)                                      \
  if (dist[b] < dist[a]) {                               \
    float x = dist[a]; dist[a] = dist[b]; dist[b] = x;   \
    uint32_t y = ids[a]; ids[a] = ids[b]; ids[b] = y;    \
  }
  RT_SW(0, 1) RT_SW(2, 3) RT_SW(0, 2) RT_SW(1, 3) RT_SW(1, 2)
#undef RT_SW
#pragma unroll
  for (int c = 3; c >= 0; --c) {
    if (dist[c] <= bound && ids[c] != EMPTY) {
      if (sp < STACK) stack[sp++] = ids[c];
      else atomicAdd(&st->stack_drops, 1ull);
    }
  }
}

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

template <class Lane>
RT_DEV void set_child(Lane& L, uint32_t child) {
  L.cur = child;
  L.phase = (child & LEAF) ? PH_LEAF : PH_NODE;
}

// ---------------------------------------------------------------- GI layout

// gi_triangle (gi_rays_software.wgsl:42-58): true with (t, u, v) inside (tmin, tmax)
RT_DEV bool gi_triangle(F3 o, F3 d, F3 a, F3 b, F3 c, float tmin, float tmax, float& t, float& u, float& v) {
  F3 e1 = sub3(b, a), e2 = sub3(c, a);
  F3 p = cross3(d, e2);
  float det = dot3(e1, p);
  if (fabsf(det) < 1e-30f) return false;
  float inv = __frcp_rn(det);
  F3 s = sub3(o, a);
  u = mul(dot3(s, p), inv);
  if (u < 0.0f || u > 1.0f) return false;
  F3 q = cross3(s, e1);
  v = mul(dot3(d, q), inv);
  if (v < 0.0f || add(u, v) > 1.0f) return false;
  t = mul(dot3(e2, q), inv);
  return t > tmin && t < tmax;
}

// unit_normal (shaders/scene.wgsl:86-90) with inverseSqrt as a correctly rounded 1/sqrt.
RT_DEV F3 unit_normal(F3 n) {
  float m = fmaxf(fmaxf(fmaxf(fabsf(n.x), fabsf(n.y)), fabsf(n.z)), 1e-30f);
  F3 s = {__fdiv_rn(n.x, m), __fdiv_rn(n.y, m), __fdiv_rn(n.z, m)};
  float k = __frcp_rn(__fsqrt_rn(fmaxf(dot3(s, s), 1e-30f)));
  return {mul(s.x, k), mul(s.y, k), mul(s.z, k)};
}

// The closest hit so far: the record's identity words and normal are made once, when the ray ends. The
// triangle is kept as a place in its mesh's index list (at most 2^32 - 1 long), not as a word of the
// buffer, which may lie past 2^32: 64 bits for it cost FAST's closest hits 1.5 % (1M GI rays over 250k
// triangles 1,087 us against 1,064).
struct GiNear {
  float t, u, v;
  uint32_t inst;  // EMPTY: none
  uint32_t at;    // the triangle's first index, in the mesh's list
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
    const size_t x = (size_t)indices + b.at;
    tri[0] = ld(w, x), tri[1] = ld(w, x + 1), tri[2] = ld(w, x + 2);
    const F3 a = ld3(w, positions + (size_t)tri[0] * 3), bb = ld3(w, positions + (size_t)tri[1] * 3),
             c = ld3(w, positions + (size_t)tri[2] * 3);
    const F3 cr = cross3(sub3(bb, a), sub3(c, a));
    const uint4 q0 = ld4(w, r), q1 = ld4(w, r + 4), q2 = ld4(w, r + 8);
    n = unit_normal({add(add(mul(__uint_as_float(q0.x), cr.x), mul(__uint_as_float(q1.x), cr.y)), mul(__uint_as_float(q2.x), cr.z)),
                     add(add(mul(__uint_as_float(q0.y), cr.x), mul(__uint_as_float(q1.y), cr.y)), mul(__uint_as_float(q2.y), cr.z)),
                     add(add(mul(__uint_as_float(q0.z), cr.x), mul(__uint_as_float(q1.z), cr.y)), mul(__uint_as_float(q2.z), cr.z))});
    if (prim_base != 0) tri[0] = ld(w, (size_t)prim_base + b.at / 3), tri[1] = 0, tri[2] = 0;
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
    const size_t x = (size_t)L.indices + first + k;  // past 2^32 where a buffer's last mesh crosses it
    const bool two = k + 3 < count;
    const size_t y = two ? x + 3 : x;
    const uint32_t ia = ld(w, x), ib = ld(w, x + 1), ic = ld(w, x + 2);
    const uint32_t ja = ld(w, y), jb = ld(w, y + 1), jc = ld(w, y + 2);
    const F3 a = ld3(w, L.positions + (size_t)ia * 3), b = ld3(w, L.positions + (size_t)ib * 3),
             c = ld3(w, L.positions + (size_t)ic * 3);
    const F3 a2 = ld3(w, L.positions + (size_t)ja * 3), b2 = ld3(w, L.positions + (size_t)jb * 3),
             c2 = ld3(w, L.positions + (size_t)jc * 3);
    float t, u, v;
    if (gi_triangle(L.o, L.d, a, b, c, L.ray.tmin, gi_limit(L.best, i), t, u, v)) {
      L.best = GiNear{t, u, v, i, first + k};
      if (any_of<AM>(L)) return true;
    }
    if (two && gi_triangle(L.o, L.d, a2, b2, c2, L.ray.tmin, gi_limit(L.best, i), t, u, v)) {
      L.best = GiNear{t, u, v, i, first + k + 3};
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

// gi_instance (gi_rays_software.wgsl:98-207) for an any-hit ray of a launch whose warps are full: true when
// something in it blocks the ray. A loop of its own, every surviving child on the stack and words loaded
// one by one: the shared steps took 2,477 us against 2,228 for 1M incoherent rays over 20 listed
// instances, 919 against 869 over one mesh, 2,163 against 1,903 for camera rays under a top level of 500
// (and 627 against 705 for 90,000 of them). Where few rays are spread over warps the wait for each load
// counts, and the shared steps, which keep the next child in a register, are ahead (300 rays over one
// mesh 76 us against 81, 20,000 under the top level 653 against 689).
RT_DEV bool gi_blocked(const uint32_t* __restrict__ w, uint32_t i, const Ray& ray, F3 world_inv, uint32_t* stack, DevStatus* st) {
  const size_t r = 16 + (size_t)i * 32;
  if ((ld(w, r + 27) & 1u) != 0) return false;
  const float lim = ray.tmax;  // nothing met yet
  if (!(slab_near(ray.o, world_inv, ld3(w, r + 12), ld3(w, r + 15), ray.tmin, lim) <= lim)) return false;
  const float r00 = ldf(w, r), r01 = ldf(w, r + 1), r02 = ldf(w, r + 2), r03 = ldf(w, r + 3);
  const float r10 = ldf(w, r + 4), r11 = ldf(w, r + 5), r12 = ldf(w, r + 6), r13 = ldf(w, r + 7);
  const float r20 = ldf(w, r + 8), r21 = ldf(w, r + 9), r22 = ldf(w, r + 10), r23 = ldf(w, r + 11);
  const F3 o = {dot4p(r00, r01, r02, r03, ray.o), dot4p(r10, r11, r12, r13, ray.o), dot4p(r20, r21, r22, r23, ray.o)};
  const F3 d = {dot3({r00, r01, r02}, ray.d), dot3({r10, r11, r12}, ray.d), dot3({r20, r21, r22}, ray.d)};
  const F3 inv = safe_inverse(d);
  const uint32_t nodes = ld(w, r + 18), leaves = ld(w, r + 19), positions = ld(w, r + 20), indices = ld(w, r + 21);
  stack[0] = ld(w, r + 22);
  uint32_t sp = 1;
  while (sp > 0) {
    const uint32_t child = stack[--sp];
    if (child & LEAF) {
      const size_t l = leaves + (size_t)(child & ~LEAF) * 2;
      const uint32_t first = ld(w, l), count = ld(w, l + 1);
      for (uint32_t k = 0; k < count; k += 6) {
        const size_t x = (size_t)indices + first + k;
        const bool two = k + 3 < count;
        const size_t y = two ? x + 3 : x;
        const uint32_t ia = ld(w, x), ib = ld(w, x + 1), ic = ld(w, x + 2);
        const uint32_t ja = ld(w, y), jb = ld(w, y + 1), jc = ld(w, y + 2);
        const F3 a = ld3(w, positions + (size_t)ia * 3), b = ld3(w, positions + (size_t)ib * 3),
                 c = ld3(w, positions + (size_t)ic * 3);
        const F3 a2 = ld3(w, positions + (size_t)ja * 3), b2 = ld3(w, positions + (size_t)jb * 3),
                 c2 = ld3(w, positions + (size_t)jc * 3);
        float t, u, v;
        if (gi_triangle(o, d, a, b, c, ray.tmin, lim, t, u, v)) return true;
        if (two && gi_triangle(o, d, a2, b2, c2, ray.tmin, lim, t, u, v)) return true;
      }
      continue;
    }
    const size_t n = nodes + (size_t)child * 16;
    const F3 oq = ld3(w, n), step = ld3(w, n + 3);
    uint32_t c[4] = {ld(w, n + 6), ld(w, n + 7), ld(w, n + 8), ld(w, n + 9)};
    const uint32_t lx = ld(w, n + 10), ly = ld(w, n + 11), lz = ld(w, n + 12);
    const uint32_t hx = ld(w, n + 13), hy = ld(w, n + 14), hz = ld(w, n + 15);
    uint32_t tb[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      tb[s] = __float_as_uint(BIG);
      if (c[s] == EMPTY) continue;
      const uint32_t sh = 8 * s;
      const F3 lo = {add(oq.x, mul(step.x, (float)((lx >> sh) & 0xffu))), add(oq.y, mul(step.y, (float)((ly >> sh) & 0xffu))),
                     add(oq.z, mul(step.z, (float)((lz >> sh) & 0xffu)))};
      const F3 hi = {add(oq.x, mul(step.x, (float)((hx >> sh) & 0xffu))), add(oq.y, mul(step.y, (float)((hy >> sh) & 0xffu))),
                     add(oq.z, mul(step.z, (float)((hz >> sh) & 0xffu)))};
      tb[s] = __float_as_uint(slab_near(o, inv, lo, hi, ray.tmin, lim));
    }
    // (distance bits, child), descending: gi_rays_software.wgsl:191-197
#define RT_SW(a, b)                          \
  if (tb[a] < tb[b]) {                       \
    uint32_t x = tb[a]; tb[a] = tb[b]; tb[b] = x; \
    x = c[a]; c[a] = c[b]; c[b] = x;         \
  }
    RT_SW(0, 1) RT_SW(2, 3) RT_SW(0, 2) RT_SW(1, 3) RT_SW(1, 2)
#undef RT_SW
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (__uint_as_float(tb[s]) <= lim && c[s] != EMPTY) {
        if (sp < STACK) stack[sp++] = c[s];
        else atomicAdd(&st->stack_drops, 1ull);
      }
    }
  }
  return false;
}

// gi_traverse (gi_rays_software.wgsl:217-279) of one ray.
template <int AM, bool SPREAD>
RT_DEV void gi_traverse(const uint32_t* __restrict__ w, GiLane<AM>& L, DevStatus* st) {
  L.world_inv = safe_inverse(L.ray.d);
  L.best = GiNear{L.ray.tmax, 0.0f, 0.0f, EMPTY, 0u};
  uint32_t stack[STACK];
  auto instance = [&](uint32_t i) {  // true when an any-hit ray is blocked
    if constexpr (AM == 1 && !SPREAD) {
      if (!gi_blocked(w, i, L.ray, L.world_inv, stack, st)) return false;
      L.best.inst = i;
      return true;
    } else {
      if (!gi_enter<AM>(w, L, i)) return false;
      for (;;) {
        uint32_t next = EMPTY;
        if (L.cur & LEAF) {
          if (gi_leaf<AM>(w, L, L.cur)) return true;
        } else {
          next = gi_node<AM>(w, L, L.cur, stack, st);
        }
        if (next == EMPTY) {
          if (L.sp == 0) return false;
          next = stack[--L.sp];
        }
        L.cur = next;
      }
    }
  };
  const uint32_t instances = ld(w, 0), top = ld(w, 1);
  if (top == 0) {
    for (uint32_t i = 0; i < instances; ++i)
      if (instance(i)) return;
    return;
  }
  uint32_t nodes[STACK];
  nodes[0] = ld(w, 2);
  uint32_t sp = 1;
  while (sp > 0) {
    const uint32_t item = nodes[--sp];
    if (item & LEAF) {
      if (instance(item & ~LEAF)) return;
      continue;
    }
    const float bound = L.best.inst != EMPTY ? next_up(L.best.t) : L.best.t;
    top_step(w, top + (size_t)item * 32, L.ray, L.world_inv, bound, nodes, sp, st);
  }
}

// Resident blocks of 128 threads an SM. Closest hits (72 registers): 6, 7 and 8 give 2.17, 2.10 and 2.15
// ms for 1M GI rays over 250k triangles, 559, 538 and 539 us for 1M camera rays there (reflection).
// Any hit (64 registers): 7, 8, 9 and 10 give 1.87, 1.76, 1.75 and 1.79 ms for 1M shadow rays there.
constexpr int PLAIN_MIN_BLOCKS = 7, PLAIN_ANY_BLOCKS = 8, PLAIN_FEW_BLOCKS = 5;  // FEW: see run_gi_closest

// The ray of this thread: `width` rays to a warp, in its first lanes (n: none).
RT_DEV uint32_t plain_ray(uint32_t width, uint32_t n) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, lane = t & 31;
  const uint64_t i = (uint64_t)(t >> 5) * width + lane;
  return lane < width && i < n ? (uint32_t)i : n;
}

// SPREAD: its warps hold few rays each.
template <int AM, class Src, int BLOCKS, bool SPREAD = false>
__global__ void __launch_bounds__(128, BLOCKS) k_gi_plain(const uint32_t* __restrict__ w, const Src src, uint32_t n, uint32_t width,
                                                          DevStatus* st) {
  const uint32_t i = plain_ray(width, n);
  if (i == n) return;
  GiLane<AM> L;
  L.ray = fetch(src, i, L);
  gi_traverse<AM, SPREAD>(w, L, st);
  gi_finish<AM>(w, L, src);
}

// ---------------------------------------------------------------- reflection layout

constexpr float RS_EDGE = 4e-6f;

struct RsBest {
  float t;
  uint32_t rec[4];
  uint32_t inst;
};

// rs_limit (reflections_software_bvh4.wgsl:45-47)
RT_DEV float rs_limit(const RsBest& b, uint32_t i) { return (b.rec[0] != 0 && i <= b.inst) ? next_up(b.t) : b.t; }

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

// rs_trace's prologue (reflections_software_bvh4.wgsl:141-155): the ray against the scene's box,
// which bounds its range; false when it misses.
template <int AM>
RT_DEV bool rs_scene(const uint32_t* __restrict__ w, size_t bounds, RsLane<AM>& L) {
  const F3 lo = ld3(w, bounds), hi = ld3(w, bounds + 4);
  const F3 o = L.ray.o, wi = L.world_inv;
  const float ax = mul(sub(lo.x, o.x), wi.x), ay = mul(sub(lo.y, o.y), wi.y), az = mul(sub(lo.z, o.z), wi.z);
  const float bx = mul(sub(hi.x, o.x), wi.x), by = mul(sub(hi.y, o.y), wi.y), bz = mul(sub(hi.z, o.z), wi.z);
  const float near = fmaxf(fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz)), L.ray.tmin);
  const float far = fminf(fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz)), L.ray.tmax);
  if (near > far) return false;
  L.best.t = fminf(L.ray.tmax, __uint_as_float(__float_as_uint(far) + 2u));
  return true;
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

// rs_trace (reflections_software_bvh4.wgsl:140-204) of one ray.
template <int AM>
RT_DEV void rs_trace(const uint32_t* __restrict__ w, RsLane<AM>& L, DevStatus* st) {
  RsBest& best = L.best;
  best.t = L.ray.tmax, best.rec[0] = best.rec[1] = best.rec[2] = best.rec[3] = 0, best.inst = EMPTY;
  L.world_inv = safe_inverse(L.ray.d);
  const uint4 head = ld4(w, 0);
  if (head.x == 0) return;
  if (!rs_scene(w, ld(w, 4) & ~3u, L)) return;
  uint32_t stack[STACK];
  auto instance = [&](uint32_t i) {  // true when an any-hit ray is blocked
    if (!rs_enter<AM>(w, L, i)) return false;
    for (;;) {
      uint32_t next = EMPTY;
      if (L.cur & LEAF) {
        if (rs_leaf<AM>(w, L, L.cur)) return true;
      } else {
        next = rs_node<AM>(w, L, L.cur, stack, st);
      }
      if (next == EMPTY) {
        if (L.sp == 0) return false;
        next = stack[--L.sp];
      }
      L.cur = next;
    }
  };
  if (head.y == 0) {
    for (uint32_t i = 0; i < head.x; ++i)
      if (instance(i)) return;
    return;
  }
  uint32_t nodes[STACK];
  nodes[0] = head.z;
  uint32_t sp = 1;
  while (sp > 0) {
    const uint32_t item = nodes[--sp];
    if (item & LEAF) {
      if (instance(item & ~LEAF)) return;
      continue;
    }
    const float bound = best.rec[0] != 0 ? next_up(best.t) : best.t;
    top_step(w, (head.y & ~3u) + (size_t)item * 32, L.ray, L.world_inv, bound, nodes, sp, st);
  }
}

template <int AM, class Src>
__global__ void __launch_bounds__(128, AM ? PLAIN_ANY_BLOCKS : PLAIN_MIN_BLOCKS) k_rs_plain(const uint32_t* __restrict__ w, const Src src, uint32_t n, uint32_t width,
                                                  DevStatus* st) {
  const uint32_t i = plain_ray(width, n);
  if (i == n) return;
  RsLane<AM> L;
  L.ray = fetch(src, i, L);
  rs_trace<AM>(w, L, st);
  rs_finish<AM>(L, src);
}

}  // namespace rtk
