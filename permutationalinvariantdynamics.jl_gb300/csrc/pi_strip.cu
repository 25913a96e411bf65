// Coefficient planes of the strip apply (pi_strip.cuh) and its launches.
#include <algorithm>

#include "../../include/picuda.h"
#include "pi_strip.cuh"
#include "pi_handle.hpp"
#include "pi_internal.hpp"

namespace picuda {
namespace {

// Strip items of sector s by the blocks of one grid row.
__device__ __forceinline__ void fill_items(const DevSector* __restrict__ sectors, int s, StripItem* __restrict__ items) {
  const DevSector& sec = sectors[s];
  const int n = sec.n;
  StripItem it{};
  it.off = (int)sec.offset;
  it.n = n;
  if (sec.src[0] >= 0) it.off0 = (int)sectors[sec.src[0]].offset, it.m0 = sectors[sec.src[0]].n;
  if (sec.src[2] >= 0) it.off2 = (int)sectors[sec.src[2]].offset, it.m2 = sectors[sec.src[2]].n;
  it.loff = sec.line0;
  it.sector = s;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; 32LL * i < (long long)n * n; i += gridDim.x * blockDim.x) {
    it.local0 = 32 * i;
    items[sec.item0 + i] = it;
  }
}

__global__ void k_strip_items(const DevSector* __restrict__ sectors, StripItem* __restrict__ items) {
  fill_items(sectors, blockIdx.y, items);
}

// Planes and line tables of sector blockIdx.y, and its strip items unless they are there, merged in FP64 for either precision.  The sums run
// over the terms in use, not the table's zero padding.
template <typename T>
__global__ void k_planes(const DevSector* __restrict__ sectors, const int4* __restrict__ canon,
                         const double2* __restrict__ coef, const StripPlanes<T> P, int nr, const TermCounts terms,
                         T* __restrict__ plane, typename Vec2<T>::type* __restrict__ lrow,
                         typename Vec2<T>::type* __restrict__ rcol, StripItem* __restrict__ items) {
  using T2 = typename Vec2<T>::type;
  const int s = blockIdx.y;
  if (items != nullptr) fill_items(sectors, s, items);
  const DevSector& sec = sectors[s];
  const int n = sec.n;
  const unsigned cnt = (unsigned)n * n;  // below 2^30, as the plan's dimension
  const int4* ct = canon + (long long)s * kCanonEntries;
  // sum of the real products at one sandwich position of the canonical table
  auto sand = [&](int pos, int a, int b) {
    double v = 0;
    for (int t = 0; t < terms.n[pos]; ++t) {
      const int4 e = ct[5 + pos * kCanonPerPos + t];
      v = fma(coef[e.x + a].x, coef[e.y + b].x, v);
    }
    return v;
  };
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
    const int b = (int)(i / (unsigned)n), a = (int)i - b * n;
    const double2 al = coef[ct[0].x + a], be = coef[ct[0].y + b];
    T* out = plane + sec.offset + i;
    out[0] = (T)((al.x + be.x) + sand(4, a, b));  // the own-sector centre gain joins the ADD term
    out[P.dim] = (T)(al.y + be.y);
    for (int k = 0; k < nr; ++k) {
      const int src = P.gain[k].src;
      const int slot = src == 0 ? 1 : src == 1 ? 0 : 2;
      out[(2 + k) * P.dim] = (T)sand(slot * 3 + P.gain[k].shift + 1, a, b);
    }
  }
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      lrow[sec.line0 + i] = T2{(T)coef[ct[1].x + i].y, (T)coef[ct[2].x + i].y};
      rcol[sec.line0 + i] = T2{(T)coef[ct[3].y + i].y, (T)coef[ct[4].y + i].y};
    }
}

// 128 columns at N = 120 with emission, dephasing and collective decay: FP64 1.41 ms = 1.21 TFLOP/s,
// 97% of the FP64 pipe (2.34 ms for 32 x 32 tiles with staged windows); FP32 200 us = 3.1 TB/s,
// bound by L1 (350 us).  37 columns at N = 97 with pumping: FP32 40 us against 75 us.  One vector
// at N = 200: FP64 62 us against 125 us, FP32 19 us against 26 us (products formed on the way).
// EPI: scale and trace border; without them their instructions are not in the kernel.
template <typename T, int V, bool EPI>
__global__ void __launch_bounds__(kStripThreads, sizeof(T) == 4 ? 8 : 4)
    k_apply_strip(const StripPlanes<T> P, const DevSector* __restrict__ sectors, int ncols, int rc,
                  const typename Vec2<T>::type* __restrict__ x, typename Vec2<T>::type* __restrict__ y, long long ld,
                  const double2* alpha, int coords, double scale) {
  using T2 = typename Vec2<T>::type;
  const int item = blockIdx.x * kStripWarps + (threadIdx.x >> 5);
  if (item >= P.nitems) return;
  const StripItem it = P.items[item];
  StripEntry<T, V> E;
  if (!E.load(it, P, threadIdx.x & 31)) return;
  const int c0 = blockIdx.y * rc, c1 = min(c0 + rc, ncols);
  x += c0 * ld;
  y += c0 * ld + E.e;
#pragma unroll 1
  for (int c = c0; c < c1; ++c) {
    T2 out = E.apply(x);
    if (EPI) {
      out.x *= (T)scale;
      out.y *= (T)scale;
      if (alpha != nullptr && E.diag) {
        const double v = coords ? sectors[it.sector].border_z : sectors[it.sector].border_x;
        const double2 al = alpha[c];
        if constexpr (sizeof(T) == 4) {
          out.x += (float)(al.x * v);
          out.y += (float)(al.y * v);
        } else {
          out.x = fma(al.x, v, out.x);
          out.y = fma(al.y, v, out.y);
        }
      }
    }
    *y = out;
    x += ld;
    y += ld;
  }
}

// Lets this thread allocate and wait while another stream of the process is being captured.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

// Records the fill that the fill stream has just been given.
static cudaError_t record_fill(pi_plan* plan, TableFill& f) {
  cudaError_t e = f.ready ? cudaSuccess : cudaEventCreateWithFlags(&f.ready, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventRecord(f.ready, plan->fill_stream);
  f.recorded = e == cudaSuccess;
  return e;
}

// Lets work that s gets from now on read the table: s waits for the fill on the GPU while it may be
// running.  A capture must not depend on work outside it, so under one the host waits instead, for
// the fill alone.  `fresh`: the fill has just been recorded.  Caller holds em_mu.
static bool order_after(TableFill& f, cudaStream_t s, bool fresh) {
  if (f.done) return true;
  RelaxedCapture relaxed;
  if (!fresh) {
    const cudaError_t q = cudaEventQuery(f.ready);
    if (q == cudaSuccess) return f.done = true;
    (void)cudaGetLastError();
    if (q != cudaErrorNotReady) return false;
  }
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone)
    return cudaStreamWaitEvent(s, f.ready, 0) == cudaSuccess;
  (void)cudaGetLastError();
  return f.done = cudaEventSynchronize(f.ready) == cudaSuccess;
}

// Device memory for a table: from the reserved room, otherwise new, an optional one within the plan's
// budget.
static char* table_alloc(pi_plan* plan, size_t bytes, bool optional = true) {
  if (char* p = plan->lazy_room.take(bytes)) return p;
  if (optional && (double)plan->device_bytes + (double)bytes > plan->memory_budget) return nullptr;
  char* p = (char*)plan_alloc(plan, bytes);
  if (!p) (void)cudaGetLastError();
  return p;
}

static size_t items_bytes(const pi_plan* plan) { return sizeof(StripItem) * (size_t)plan->nstrip_items; }

// 32-bit element indices within a vector
static bool has_items(const DevicePlan& dp) { return dp.dim > 0 && dp.dim <= 0x3fffffffLL; }

static bool items_memory(pi_plan* plan, bool optional) {
  if (!plan->items_mem) plan->items_mem = (StripItem*)table_alloc(plan, items_bytes(plan), optional);
  return plan->items_mem != nullptr;
}

StripItems strip_items(pi_plan* plan, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(plan->em_mu);
  const DevicePlan& dp = plan->dev;
  const bool fresh = !plan->items_fill.recorded;
  if (fresh) {
    RelaxedCapture relaxed;
    if (!plan->strip_items) {
      if (!has_items(dp)) return StripItems{};
      // An FP32 step by strips needs them beside its split planes, which have no budget either: by
      // tiles from the general terms it would round differently from the persistent schedules.
      if (!items_memory(plan, false)) return StripItems{};
      k_strip_items<<<dim3(8, (unsigned)dp.nsectors), 256, 0, plan->fill_stream>>>(dp.sectors, plan->items_mem);
      if (cudaGetLastError() != cudaSuccess) return StripItems{};
      plan->strip_items = plan->items_mem;
    }
    if (record_fill(plan, plan->items_fill) != cudaSuccess) return StripItems{};
  }
  if (!order_after(plan->items_fill, s, fresh)) return StripItems{};
  return StripItems{plan->strip_items, plan->nstrip_items};
}

// Line tables and planes of one precision: [row shifts][column shifts][2 + nr planes].
template <typename T>
struct PlaneBytes {
  size_t line, all;
  PlaneBytes(const pi_plan* plan, int nr)
      : line((2 * sizeof(T) * (size_t)plan->nlines + 15) / 16 * 16),
        all(2 * line + (sizeof(T) * (size_t)plan->dev.dim * (2 + nr) + 15) / 16 * 16) {}
};

// Gain positions that some sector uses, in the order of the canonical kernels: own, smaller, larger
// sector.  Returns their number; *drive: some sector has line shifts.
static int gain_positions(const pi_plan* plan, GainPos (&gain)[kMaxGains], bool* drive) {
  bool used[3][3] = {};
  *drive = false;
  for (const Sector& sec : plan->host.sectors)
    for (const StencilTerm& t : sec.terms) {
      *drive = *drive || t.kind == ST_LEFT || t.kind == ST_RIGHT;
      if (t.kind == ST_SAND) used[t.e == 0 ? 0 : t.e < 0 ? 1 : 2][t.p + 1] = true;
    }
  used[0][1] = false;  // joins the centre
  for (GainPos& g : gain) g = GainPos{-1, 0};
  int nr = 0;
  for (int src = 0; src < 3; ++src)
    for (int p = -1; p <= 1; ++p)
      if (used[src][p + 1]) gain[nr++] = GainPos{(signed char)src, (signed char)p};
  return nr;
}

size_t reserve_bytes(const pi_plan* plan) {
  if (!has_items(plan->dev)) return 0;
  GainPos gain[kMaxGains];
  bool drive;
  const int nr = gain_positions(plan, gain, &drive);
  return TableRoom::padded(items_bytes(plan)) + TableRoom::padded(PlaneBytes<double>(plan, nr).all);
}

// Room for the items and the first FP64 planes (or FP32 ones of both coordinate systems).  The
// allocation is a small part of compile(), and most of a first apply that has to make it: 0.17 ms
// of 0.34 at N = 200, where compile() takes 78.  Small plans have the room at the end of their
// tables' allocation.
void reserve_planes(pi_plan* plan) {
  const size_t bytes = plan->dev.canon ? reserve_bytes(plan) : 0;
  if (bytes == 0 || plan->lazy_room.base || plan->strip_items) return;
  if ((double)plan->device_bytes + (double)bytes > plan->memory_budget) return;
  if (char* p = plan->own_room.take(bytes)) {
    plan->lazy_room = TableRoom{p, bytes, 0};
    plan->device_bytes += bytes;
  } else {
    plan->lazy_room.base = (char*)plan_alloc(plan, bytes);
    if (!plan->lazy_room.base) return (void)cudaGetLastError();
    plan->lazy_room.size = bytes;
    list_reserve(plan);
  }
  for (TableFill* f : {&plan->planes64_fill[0], &plan->planes32_fill[0]})  // a first apply's only event
    if (cudaEventCreateWithFlags(&f->ready, cudaEventDisableTiming) != cudaSuccess) (void)cudaGetLastError();
}

template <typename T>
static StripPlanes<T> build_planes(pi_plan* plan, int coords, cudaStream_t s, StripPlanes<T> (&kept)[2],
                                   TableFill (&fill)[2], bool (&failed)[2]) {
  using T2 = typename Vec2<T>::type;
  const DevicePlan& dp = plan->dev;
  if (!dp.canon) return StripPlanes<T>{};
  std::lock_guard<std::recursive_mutex> lk(plan->em_mu);
  const int which = coords ? 1 : 0;
  StripPlanes<T>& P = kept[which];
  if (P.items) return order_after(fill[which], s, false) ? P : StripPlanes<T>{};
  if (failed[which] || !has_items(dp)) return StripPlanes<T>{};
  RelaxedCapture relaxed;
  StripPlanes<T> Q;
  Q.dim = dp.dim;
  Q.nitems = plan->nstrip_items;
  bool drive;
  const int nr = gain_positions(plan, Q.gain, &drive);
  Q.variant = drive ? (nr <= 1 ? 0 : nr <= 3 ? 1 : nr <= 5 ? 2 : nr <= 6 ? 3 : 4) : (nr <= 5 ? 5 : 6);
  const PlaneBytes<T> bytes(plan, nr);
  char* d = items_memory(plan, true) ? table_alloc(plan, bytes.all) : nullptr;
  failed[which] = d == nullptr;  // no room: the plan keeps the general kernels
  if (!d) return StripPlanes<T>{};
  Q.items = plan->items_mem;
  Q.lrow = (const T2*)d;
  Q.rcol = (const T2*)(d + bytes.line);
  Q.plane = (const T*)(d + 2 * bytes.line);
  const dim3 grid((unsigned)std::min<long long>(64, ((long long)plan->host.max_n * plan->host.max_n + 255) / 256),
                  (unsigned)dp.nsectors);
  // behind items filled before on the same stream, so its event covers them
  k_planes<T><<<grid, 256, 0, plan->fill_stream>>>(dp.sectors, dp.canon, coords ? dp.coef64z : dp.coef64, Q, nr,
                                                   dp.canon_terms, (T*)Q.plane, (T2*)Q.lrow, (T2*)Q.rcol,
                                                   plan->strip_items ? nullptr : plan->items_mem);
  if (cudaGetLastError() != cudaSuccess || record_fill(plan, fill[which]) != cudaSuccess) {
    failed[which] = true;
    return StripPlanes<T>{};
  }
  plan->strip_items = plan->items_mem;
  P = Q;
  return order_after(fill[which], s, true) ? P : StripPlanes<T>{};
}

Planes64 planes64(pi_plan* plan, int coords, cudaStream_t s) {
  return build_planes<double>(plan, coords, s, plan->planes64, plan->planes64_fill, plan->planes64_failed);
}

Planes32 planes32(pi_plan* plan, int coords, cudaStream_t s) {
  return build_planes<float>(plan, coords, s, plan->planes32, plan->planes32_fill, plan->planes32_failed);
}

namespace {

template <typename T, int V>
void launch_variant(const dim3 grid, cudaStream_t stream, const StripPlanes<T>& P, const DevicePlan& dp, int ncols,
                    int rc, const T* x, T* y, long long ld, const BorderArgs& border) {
  using T2 = typename Vec2<T>::type;
  const bool epi = border.scale != 1.0 || border.alpha != nullptr;
  auto k = epi ? k_apply_strip<T, V, true> : k_apply_strip<T, V, false>;
  k<<<grid, kStripThreads, 0, stream>>>(P, dp.sectors, ncols, rc, (const T2*)x, (T2*)y, ld, border.alpha,
                                        border.coords, border.scale);
}

}  // namespace

template <typename T>
cudaError_t launch_apply_strip(const DevicePlan& dp, const StripPlanes<T>& P, const T* x, T* y, int ncols,
                               long long ld, const BorderArgs& border, cudaStream_t s) {
  // Columns per block: an entry's coefficients are about as many loads as a column's sources, so
  // up to 16 columns share them while two waves of warps remain.  FP32, 37 columns at N = 97 (two
  // to 32 per block): 55, 44, 41, 40, 48 us; 128 at N = 120: 302, 240, 212, 203, 199 us.
  int rc = 16;
  while (rc > 1 && (long long)P.nitems * ((ncols + rc - 1) / rc) < 2LL * 152 * 32) rc /= 2;
  const dim3 grid((unsigned)((P.nitems + kStripWarps - 1) / kStripWarps), (unsigned)((ncols + rc - 1) / rc));
  static_assert(kStripVariants == 7, "one launch per variant");
  switch (P.variant) {
    case 0: launch_variant<T, 0>(grid, s, P, dp, ncols, rc, x, y, ld, border); break;
    case 1: launch_variant<T, 1>(grid, s, P, dp, ncols, rc, x, y, ld, border); break;
    case 2: launch_variant<T, 2>(grid, s, P, dp, ncols, rc, x, y, ld, border); break;
    case 3: launch_variant<T, 3>(grid, s, P, dp, ncols, rc, x, y, ld, border); break;
    case 4: launch_variant<T, 4>(grid, s, P, dp, ncols, rc, x, y, ld, border); break;
    case 5: launch_variant<T, 5>(grid, s, P, dp, ncols, rc, x, y, ld, border); break;
    default: launch_variant<T, 6>(grid, s, P, dp, ncols, rc, x, y, ld, border);
  }
  return cudaGetLastError();
}

template cudaError_t launch_apply_strip<double>(const DevicePlan&, const Planes64&, const double*, double*, int,
                                                long long, const BorderArgs&, cudaStream_t);
template cudaError_t launch_apply_strip<float>(const DevicePlan&, const Planes32&, const float*, float*, int,
                                               long long, const BorderArgs&, cudaStream_t);

}  // namespace picuda
