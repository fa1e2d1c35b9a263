// Internal state behind the C ABI's opaque handles, shared by the translation units that
// implement it (rt_api.cu, batches.cu).
#pragma once
#include <cuda_runtime.h>

#include <array>
#include <atomic>
#include <cstdarg>
#include <map>
#include <vector>
#include <cstdio>
#include <mutex>
#include <string>

#include "../../include/rt_trace.h"
#include "host/host.hpp"
#include "host/wide8.hpp"
#include "launch.hpp"

// Per BLAS of a scene, what rt_scene_refit needs about its (fixed) topology.
struct RefitLevels {
  uint32_t node_count = 0;
  uint32_t tri_count = 0;       // reflection layout: packed triangles of the BLAS
  uint32_t position_count = 0;  // GI layout: position records of the BLAS
  uint32_t* d_tree = nullptr;   // per node: its parent, a counter, and (bytes) its inner children
  // Instead, where the nodes are not one tree: d_tree holds node ids by height above the leaves, height
  // h at [level_start[h], level_start[h + 1]).
  std::vector<uint32_t> level_start;
};

struct rt_scene {
  uint32_t layout = 0;
  uint32_t* d_words = nullptr;
  size_t n_words = 0;
  rtb::SceneInfo info;
  uint32_t head[8] = {};  // the header's first words, as they are on the device
  std::vector<uint32_t> blas_words;  // words 18-23 of each instance record: its BLAS (rt_scene_refit reads them here)
  size_t device_bytes = 0;
  void* d_wide8 = nullptr;
  size_t wide8_bytes = 0;
  size_t w8_nodes_at = 0, w8_tris_at = 0, w8_inst_at = 0;
  uint32_t w8_depth = 0;  // levels of the deepest 8-wide BLAS
  // The WIDE8 walk's 8-wide top level over the instance world boxes (its own allocation: nodes,
  // then instance items). Built by rt_scene_prepare when the packed scene has a top level; a
  // rewrite of the records or the top level makes it stale, and the walk then uses the packed
  // BVH4 top level until rt_scene_prepare builds it again.
  void* d_w8_top = nullptr;
  size_t w8_top_bytes = 0, w8_top_items_at = 0;
  uint32_t w8_top_nodes = 0;
  bool w8_top_valid = false;
  uint32_t w8_entries = 0;  // the top level's entries per instance (rt_scene_tune_top); 0: the context's

  std::map<std::array<uint32_t, 4>, RefitLevels> refit;  // by the words that name the BLAS's parts (see blas_of)
  // rt_scene_move_instances: staging for the moved instances and mesh boxes, and the top level's
  // links (see k_refit_top), made by the first move and by each rebuild.
  std::vector<char> move_stage;
  void* d_move = nullptr;
  size_t move_bytes = 0;
  uint32_t* d_top_tree = nullptr;
  size_t top_cap = 0;      // nodes d_top_tree has room for
  uint32_t top_nodes = 0;  // nodes the links cover; 0: not made yet

  // rt_scene_move_instances and rt_scene_refit return with their work queued on the caller's stream
  // (see after_changes): `changed` is recorded after the last of it, on the stream with the id
  // `change_stream`; `changes` counts such calls and `settled` is the last of them known to be over.
  // `legacy` orders a change after the default stream's work.
  cudaEvent_t changed = nullptr, legacy = nullptr;
  std::atomic<unsigned long long> change_stream{0};
  std::atomic<uint64_t> changes{0};
  mutable std::atomic<uint64_t> settled{0};
};

struct rt_blas {
  rtb::Blas b;
};

struct rt_rnf {
  rtb::Rnf f;
};

// Chunks a host-buffer call keeps in flight, each with its own stream and staging slot. A
// stream runs its chunk's copy in, trace and copy out in order, so with two slots the next copy
// in waits for the copy out two chunks back; four leave the copies off the critical path.
#ifndef RT_HOST_STAGES
#define RT_HOST_STAGES 4
#endif

// Bytes of each BLAS build workspace that a context keeps (meshes of about 300k triangles) until
// rt_ctx_trim, a server on the context, an allocation that finds no room, or its end.
constexpr size_t BUILD_KEEP = 64u << 20;

struct rt_ctx {
  int device = 0;
  rtk::DevStatus* d_status = nullptr;
  uint32_t* d_scratch = nullptr;  // 16 words for the self-test
  // Ray counters of persistent launches: launch k uses slot k mod COUNTER_SLOTS, so up to that
  // many launches may be in flight at once across streams.
  unsigned int* d_counters = nullptr;
  std::atomic<uint64_t> counter_seq{0};
  rt_tuning tuning = {8, 8, RT_STACK_LOCAL, rtb::W8_BRAID_PER_INSTANCE, {0, 0, 0, 0}};
  bool stack_chosen = false;  // rt_ctx_set_tuning has named a stack placement
  std::mutex mu;
  std::string last_error;
  std::atomic<uint64_t> rays{0}, launches{0}, scene_bytes{0};
  // rt_trace_host staging: HOST_STAGES chunks in flight, one stream and staging slot each.
  cudaStream_t streams[RT_HOST_STAGES] = {};
  void* d_rays = nullptr;
  void* d_hits = nullptr;
  size_t stage_rays = 0;  // rays per chunk buffer
  // rt_order_rays scratch
  void* d_order_scratch = nullptr;
  size_t order_scratch_bytes = 0;
  // rt_blas_build_device's two workspaces, kept up to BUILD_KEEP bytes each (under `mu`)
  struct Space {
    void* p = nullptr;
    size_t bytes = 0;
  } build_space[2];
  // rt_trace_batches: batch tables staged through a ring of pinned / device slots, each reused
  // once the copy that last read it has completed.
  static constexpr uint32_t TABLE_SLOTS = 8;
  rtk::BatchEntry* h_tables = nullptr;
  rtk::BatchEntry* d_tables = nullptr;
  cudaEvent_t table_done[TABLE_SLOTS] = {};
  uint32_t table_seq = 0;
};

namespace rtc {

// The instance top level built on the device (tlas_build.cu), word for word rtb::tlas_build's:
// instance i's box is lo xyz at d_box_words[i * stride], hi xyz right after (float bits). The
// nodes go to d_out (cap_words available, the rest zeroed). Synchronous
// on `st`; the caller holds the context's lock.
rt_status tlas_build_device(rt_ctx* ctx, const uint32_t* d_box_words, size_t stride, uint32_t n, bool sah, uint32_t* d_out,
                            size_t cap_words, uint32_t* n_nodes,
                            cudaStream_t st);

constexpr size_t GI_HIT_BYTES = 40, RS_HIT_BYTES = 20, ANY_HIT_BYTES = 4, RAY_BYTES = 32;
#ifndef RT_HOST_CHUNK_LOG2
#define RT_HOST_CHUNK_LOG2 20
#endif
// Rays a host-buffer call stages per chunk (copies of one chunk overlap the next chunk's kernel).
// 2^20: measured end to end on the precision-4M step (16.8M rays, four stages) at 771 Mrays/s,
// against 752 for 2^19 (more launches, each with its tail of idle lanes and its final pass) and
// 773 for 2^21 (eight stages of 2^20: 776).
constexpr uint32_t HOST_CHUNK = 1u << RT_HOST_CHUNK_LOG2;
constexpr uint32_t HOST_CHUNK_LEAST = 1u << 18;  // rays of a chunk of a smaller call
constexpr uint32_t COUNTER_SLOTS = 4096;

inline rt_status fail(rt_ctx* ctx, rt_status s, const char* fmt, ...) {
  if (ctx) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    ctx->last_error = buf;
  }
  return s;
}

#define RT_CUDA(ctx, call)                                                                     \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) return fail(ctx, RT_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

// Event calls about work outside any stream capture, also while this thread captures.
class OutsideCapture {
 public:
  OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  ~OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }

 private:
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// The host waits for the scene's last move or refit. For the calls that read or write the scene's
// words by synchronous copies, which wait for no non-blocking stream.
inline cudaError_t wait_changes(const rt_scene* scene) {
  const uint64_t n = scene->changes.load(std::memory_order_acquire);
  if (scene->settled.load(std::memory_order_relaxed) >= n) return cudaSuccess;
  OutsideCapture guard;
  const cudaError_t e = cudaEventSynchronize(scene->changed);
  if (e == cudaSuccess) scene->settled.store(n, std::memory_order_relaxed);
  return e;
}

// after_changes on a stream, with this id, that does not capture; `n`: the changes so far.
inline cudaError_t after_changes_on(const rt_scene* scene, cudaStream_t s, unsigned long long id, uint64_t n) {
  if (id == scene->change_stream.load(std::memory_order_relaxed)) return cudaSuccess;  // in the stream's own order
  OutsideCapture guard;
  const cudaError_t e = cudaEventQuery(scene->changed);
  if (e == cudaSuccess) scene->settled.store(n, std::memory_order_relaxed);
  if (e != cudaErrorNotReady) return e;
  cudaGetLastError();
  return cudaStreamWaitEvent(s, scene->changed, 0);
}

// What is queued on `s` from here on runs after the scene's last move or refit, whichever stream that
// took: every launch that reads the scene's words is ordered so. A launch being captured runs
// later, on any stream, so there the host waits. Once the change is known to be over, two loads.
inline cudaError_t after_changes(const rt_scene* scene, cudaStream_t s) {
  const uint64_t n = scene->changes.load(std::memory_order_acquire);
  if (scene->settled.load(std::memory_order_relaxed) >= n) return cudaSuccess;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &status) != cudaSuccess || status != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return wait_changes(scene);
  }
  unsigned long long id = 0;
  const cudaError_t e = cudaStreamGetId(s, &id);
  return e != cudaSuccess ? e : after_changes_on(scene, s, id, n);
}

// Around the launches that change a scene's words on `s` (the caller holds the context's lock):
// start(), on a stream that does not capture, queues them after earlier changes and after the default
// stream's work (a traversal there that still reads the words), and the end of the scope marks them as the last change, on every
// return path.
class Change {
 public:
  Change(rt_scene* scene, cudaStream_t s) : scene_(scene), s_(s) {}
  Change(const Change&) = delete;
  Change& operator=(const Change&) = delete;
  cudaError_t start() {
    for (cudaEvent_t* ev : {&scene_->changed, &scene_->legacy})
      if (!*ev) {
        const cudaError_t e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
      }
    cudaError_t e = cudaStreamGetId(s_, &id_);
    const uint64_t n = scene_->changes.load(std::memory_order_relaxed);
    if (e == cudaSuccess && scene_->settled.load(std::memory_order_relaxed) < n) e = after_changes_on(scene_, s_, id_, n);
    if (e == cudaSuccess && s_ != nullptr && s_ != cudaStreamLegacy) {
      e = cudaEventRecord(scene_->legacy, cudaStreamLegacy);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(s_, scene_->legacy, 0);
    }
    started_ = e == cudaSuccess;
    return e;
  }
  ~Change() {
    if (!started_) return;
    cudaEventRecord(scene_->changed, s_);
    scene_->change_stream.store(id_, std::memory_order_relaxed);
    scene_->changes.fetch_add(1, std::memory_order_release);
  }

 private:
  rt_scene* scene_;
  cudaStream_t s_;
  unsigned long long id_ = 0;
  bool started_ = false;
};

// Gives the kept build workspaces back (no build runs: the caller holds the context's lock, as a build
// does throughout). Returns their bytes.
inline size_t drop_build_space(rt_ctx* ctx) {
  size_t bytes = 0;
  for (auto& b : ctx->build_space) {
    cudaFree(b.p);
    bytes += b.bytes;
    b.p = nullptr, b.bytes = 0;
  }
  return bytes;
}

// cudaMalloc for what a caller asks for: where the device has no room, again without the kept build
// workspaces. `held`: the caller holds the context's lock.
template <class T>
cudaError_t device_alloc(rt_ctx* ctx, T** p, size_t bytes, bool held = false) {
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  std::unique_lock<std::mutex> lock(ctx->mu, std::defer_lock);
  if (!held) lock.lock();
  if (drop_build_space(ctx) == 0) return e;
  cudaGetLastError();
  return cudaMalloc(reinterpret_cast<void**>(p), bytes);
}

inline size_t hit_bytes(uint32_t layout, uint32_t mode) {
  if (mode != 0) return ANY_HIT_BYTES;
  return layout == 0 ? GI_HIT_BYTES : RS_HIT_BYTES;
}

inline rtl::SceneView view_of(const rt_scene* s) {
  rtl::SceneView v;
  v.layout = s->layout;
  v.words = s->d_words;
  v.n_words = s->n_words;
  v.instances = s->info.instances;
  v.top = s->info.top;
  v.wide8 = s->d_wide8;
  v.wide8_bytes = s->wide8_bytes;
  v.w8_nodes_at = s->w8_nodes_at, v.w8_tris_at = s->w8_tris_at, v.w8_inst_at = s->w8_inst_at;
  v.w8_depth = s->w8_depth;
  v.w8_top = s->w8_top_valid ? s->d_w8_top : nullptr;
  v.w8_top_nodes = s->w8_top_valid ? s->w8_top_nodes : 0;
  v.w8_top_items_at = s->w8_top_items_at;
  return v;
}

// The stack placement that the caller has chosen for the WIDE8 per-ray walk (0: none).
inline uint32_t chosen_stack(const rt_ctx* ctx) { return ctx->stack_chosen ? ctx->tuning.wide8_stack : 0u; }
// 1 for the shared stack, 0 for the local one: the choice where there is one, else shared for any-hit
// launches over flat scenes whose trees fit it (0.84M shadow rays over 250k triangles 621 against 648
// us; closest hits there 4.68 against 4.67 ms, and over a top level 7.56 against 7.32).
inline uint32_t stack_of(uint32_t chosen, const rtl::SceneView& v, bool any_hit) {
  if (chosen) return chosen == RT_STACK_SHARED ? 1u : 0u;
  return any_hit && v.top == 0 && rtl::shared_stack_fits(v) ? 1u : 0u;
}

}  // namespace rtc
