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
// its triangle is, and the record is made when the ray ends. Together, before and after (us; the first two
// by perf/cases.py, whose scenes differ by seed: the counters above are of another seed):
//   gather of 16,384 cells over 400 instances, closest          12,288 -> 7,319
//   16,384 cells x 40 lights, 250k triangles, any hit              533 ->   450
//   1M rays, uniform directions, 250k cluster triangles, closest, GI / reflection  1,531 / 1,188 -> 1,066 / 837
//   1M camera rays, the same scene                               1,053 /   811 ->   768 / 614
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

// ---------------------------------------------------------------- reflection layout

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
      const bool live = head.x != 0 && rs_scene(w, bounds, L);
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
