// The opaque pi_plan handle behind the C ABI.
#pragma once

#include <atomic>
#include <limits>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "pi_internal.hpp"
#include "pi_plan.hpp"

namespace picuda {
class Engine;

// A device buffer that tables are cut from, at 256-byte boundaries.
struct TableRoom {
  char* base = nullptr;
  size_t size = 0, used = 0;
  static size_t padded(size_t bytes) { return (bytes + 255) / 256 * 256; }
  char* take(size_t bytes) {  // null when there is no room left
    if (used + padded(bytes) > size) return nullptr;
    char* p = base + used;
    used += padded(bytes);
    return p;
  }
};

// A table that is filled on the plan's fill stream: `ready` is recorded behind the fill, `done` once
// it is known to have passed.
struct TableFill {
  cudaEvent_t ready = nullptr;
  bool recorded = false, done = false;
};
}  // namespace picuda

struct pi_plan {
  picuda::QubitPlan host;
  picuda::DevicePlan dev;
  std::vector<void*> allocations;  // device buffers owned by the plan tables
  picuda::TableRoom own_room;      // the tables that the plan is made with
  bool reserves = false;           // pi_plan_set_memory_budget has been called
  picuda::TableRoom lazy_room;     // reserved for those that first applies lay out (guarded by em_mu)
  size_t device_bytes = 0;
  double memory_budget = std::numeric_limits<double>::infinity();  // of device_bytes, for optional tables
  long long stencil_terms = 0;
  cudaStream_t stream = nullptr;
  int device = 0;
  picuda::ReduceScratch rs;        // reduction scratch (device)
  double* host_pinned = nullptr;   // small pinned staging buffer for reductions
  // Host-buffer applies: grow-only device staging and copy/compute pipeline streams.
  void* stage_x = nullptr;
  void* stage_y = nullptr;
  size_t stage_bytes = 0;
  cudaStream_t pipe[3] = {nullptr, nullptr, nullptr};
  // Calls that use the plan's stream, staging buffers or engine hold call_mu.  By default a
  // second caller waits (the locked MatrixFreeLiouvillian of liouvillian.jl:35-60); with
  // reject_concurrent set it gets PI_ERR_BUSY instead (the workspace rule of
  // threaded_apply.jl:575).  Recursive, like the reference's ReentrantLock.
  std::recursive_mutex call_mu;
  std::atomic<int> reject_concurrent{0};
  // Element-major batched apply (pi_apply_em.cu): tile list and merged coefficient planes,
  // built on first use (FP32 reference / population coordinates).
  std::recursive_mutex em_mu;  // recursive: an allocation under it may reclaim this plan's reserve
  const picuda::DevTile* em_tiles = nullptr;
  int em_ntiles = 0;
  const float2* em_planes32[2] = {nullptr, nullptr};
  // Encoded per-sector TMA tensor maps of the last few element-major source batches (host
  // copies, passed to the kernel by value), keyed by source pointer, stride, width and right-hand
  // sides per box.  An apply in another thread may displace a set that this one is about to
  // launch with, so a set lives as long as somebody holds it.
  using EmMapBlob = std::shared_ptr<const std::vector<unsigned char>>;  // nsectors x 128 bytes
  struct EmMapSet {
    const void* x;
    long long ld;
    int ncols, g;  // width, right-hand sides per box
    EmMapBlob maps;
  };
  std::vector<EmMapSet> em_maps;
  // Split coefficient planes of the TMA-staged kernel (entry, row and column planes) per
  // coordinate system.
  struct EmSplit {
    const float4* eplane = nullptr;
    const float4* lrow = nullptr;
    const float4* rcol = nullptr;
    const float4* srow = nullptr;  // separable line planes of the single-column tile apply
    const float4* scol = nullptr;
  };
  EmSplit em_split[2];
  const void* em_tma_tiles[3][3] = {};  // tile records: 16 / 32 / 64 rows x 8 / 16 / 32 columns
  int em_tma_ntiles[3][3] = {};
  // Element-major kernel chosen by the autotuner (or pinned by the caller) per batch width
  // and coordinate system: kind 0 TMA-staged with tiles of `rows` rows and blocks of g right-hand
  // sides, 1 plain loads.
  struct EmChoice {
    int ncols, coords, kind, rows;
    double ms;  // timed duration of one apply (0 when pinned)
    int g = 64;
  };
  std::vector<EmChoice> em_choices;
  std::mutex em_tune_mu;
  // Strip items and merged coefficient planes per coordinate system, built on first use (guarded by
  // em_mu); a plan without room for them, in memory or in its budget, keeps the general kernels.
  // They are filled on a stream of their own, on which nothing else runs: a first apply waits on
  // the GPU for the fill only, not for the solves that `stream` has queued.
  cudaStream_t fill_stream = nullptr;
  picuda::StripItem* items_mem = nullptr;
  const picuda::StripItem* strip_items = nullptr;  // items_mem once its fill is queued
  int nstrip_items = 0, nlines = 0;
  picuda::Planes64 planes64[2];
  picuda::Planes32 planes32[2];
  picuda::TableFill items_fill, planes64_fill[2], planes32_fill[2];
  bool planes64_failed[2] = {false, false};
  bool planes32_failed[2] = {false, false};
  // Single-instance solves run as one job of a batched engine kept with the plan (created on
  // first use for a Krylov dimension and basis precision, replaced when those change).
  picuda::Engine* engine = nullptr;
  int engine_m = 0;
  bool engine_f32 = false;
};

namespace picuda {

// Thread-local error message for pi_last_error.
void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

// RAII guard around one call on a plan: waits for the plan's other callers (default), or,
// when the plan was switched to rejection, fails at once (ok = false) while another thread
// holds it.
struct BusyGuard {
  pi_plan* p;
  bool ok;
  explicit BusyGuard(pi_plan* plan) : p(plan) {
    if (p->reject_concurrent.load()) {
      ok = p->call_mu.try_lock();
    } else {
      p->call_mu.lock();
      ok = true;
    }
  }
  ~BusyGuard() {
    if (ok) p->call_mu.unlock();
  }
};

// Device allocation tracked by the plan; returns nullptr on failure.
void* plan_alloc(pi_plan* plan, size_t bytes);

// Reserves device memory for the strip items and the first merged coefficient planes of a canonical
// plan, as far as its budget lets it (pi_strip.cu).  What a plan has reserved and not used is given
// back when an allocation fails: reclaim_reserves() frees it on every listed plan and says whether
// there was any.
void reserve_planes(pi_plan* plan);
size_t reserve_bytes(const pi_plan* plan);  // what that takes on a canonical plan
void list_reserve(pi_plan* plan);
bool reclaim_reserves();

// Split coefficient planes of a canonical plan in reference (which 0) or population (which 1)
// FP32 coordinates, built on first use (pi_apply_em.cu); PI_ERR_UNSUPPORTED for a plan whose
// stencil does not sit at the canonical positions.
int em_split_planes(pi_plan* plan, int which, SplitPlanes* out);

// Strip items of a plan (32 consecutive entries of one sector block each), built on first use;
// items == nullptr without room for them.  Work that stream s gets after the call may read them.
struct StripItems {
  const StripItem* items = nullptr;
  int n = 0;
};
StripItems strip_items(pi_plan* plan, cudaStream_t s);

// Merged coefficient planes of a canonical plan in reference (coords 0) or population (1)
// coordinates, built on first use (pi_strip.cu), for work that stream s gets after the call;
// items == nullptr when the plan is not canonical or has no room for them.
Planes64 planes64(pi_plan* plan, int coords, cudaStream_t s);
Planes32 planes32(pi_plan* plan, int coords, cudaStream_t s);

}  // namespace picuda
