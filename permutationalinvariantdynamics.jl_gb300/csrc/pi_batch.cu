// Multi-instance Krylov engine (see pi_batch.hpp): device kernels over the engine's
// (instance, tile) and (instance, chunk) work lists, the engine's stage execution, the
// dynamics and steady-state job controllers, and the batched C entry points.
#include "pi_batch.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <exception>
#include <map>
#include <mutex>
#include <random>
#include <system_error>
#include <thread>
#include <tuple>
#include <type_traits>
#include <unordered_set>
#include <utility>

#include "pi_strip.cuh"
#include "pi_apply_impl.cuh"
#include "pi_dense.hpp"
#include "pi_reduce.cuh"

namespace picuda {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }

__device__ __forceinline__ double2 ld2(const double2* p) { return *p; }
__device__ __forceinline__ double2 ld2(const float2* p) {
  const float2 v = *p;
  return make_double2((double)v.x, (double)v.y);
}
__device__ __forceinline__ void st2(double2* p, double x, double y) { *p = make_double2(x, y); }
__device__ __forceinline__ void st2(float2* p, double x, double y) { *p = make_float2((float)x, (float)y); }

constexpr int kRT = kReduceThreads;  // threads of the chunk kernels

// Deterministic block sum of NV values (blockDim.x a multiple of 32); result in thread 0.  Warps
// from `nw` on hold zeros and stay off the FP64 pipe; the sum is the same.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* smem, int nw = kRT / 32) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < nw) {
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
  }
  if (nw == 1) {  // uniform
    __syncthreads();
    return;
  }
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) smem[warp * NV + k] = v[k];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = lane < nw ? smem[lane * NV + k] : 0.0;
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
  }
}

__device__ __forceinline__ void chunk_range(const DevInst& S, int c, long long& beg, long long& end) {
  beg = (long long)(c - S.chunk_begin) * S.chunk;
  end = min(beg + (long long)S.chunk, S.dim);
}


// ---------------------------------------------------------------------------------------
// Stage-1 kernels
// ---------------------------------------------------------------------------------------

// Norm partial of a combination whose result is the vector to be normed (dynamics trials): the
// chunk's |cout|^2 into part, as k_s1_norm_partial would leave it.
__device__ __forceinline__ void combined_norm(const DevInst& S, double v, double* part) {
  __shared__ double smem[kRT / 32];
  if (S.nrm0 != S.cout) return;  // block-uniform
  double acc[1] = {v};
  block_sum<1>(acc, smem);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = acc[0];
    part[2 * blockIdx.x + 1] = 0.0;
  }
}

// cout (+)= sum_k ccoef[k] V_k, FP64 accumulation.
__global__ void __launch_bounds__(kRT)
    k_s1_combine(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst, double* __restrict__ part) {
  __shared__ double2 cs[kBatchMaxKrylov + 2];
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  double2* out = S.cout;
  if (!out) return;
  const int nc = S.ccount;
  for (int i = threadIdx.x; i < nc; i += blockDim.x) cs[i] = S.ccoef[i];
  __syncthreads();
  long long beg, end;
  chunk_range(S, blockIdx.x, beg, end);
  const double2* V = (const double2*)S.V;
  const long long ld = S.ldv;
  const int acc = S.cacc;
  double nrm = 0;
  for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
    double yx = 0, yy = 0;
#pragma unroll 8
    for (int k = 0; k < nc; ++k) {
      const double2 v = V[(long long)k * ld + e];
      yx = fma(v.x, cs[k].x, yx);
      yx = fma(-v.y, cs[k].y, yx);
      yy = fma(v.x, cs[k].y, yy);
      yy = fma(v.y, cs[k].x, yy);
    }
    if (acc) {
      const double2 o = out[e];
      yx += o.x;
      yy += o.y;
    }
    out[e] = make_double2(yx, yy);
    nrm = fma(yy, yy, fma(yx, yx, nrm));
  }
  combined_norm(S, nrm, part);
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

// Complex normal probe (unit variance): Box-Muller on a counter-based 64-bit hash
// (SplitMix64 finaliser) of (seed, element).
__global__ void __launch_bounds__(kRT) k_s1_probe(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst) {
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  double2* p = S.probe;
  if (!p) return;
  long long beg, end;
  chunk_range(S, blockIdx.x, beg, end);
  const unsigned long long seed = mix64(S.seed);
  for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
    const unsigned long long h = mix64(seed ^ (unsigned long long)e);
    const double u1 = ((double)(h >> 32) + 1.0) * 2.3283064365386963e-10;  // (0, 1]
    const double u2 = (double)(h & 0xffffffffULL) * 2.3283064365386963e-10;  // [0, 1)
    const double r = sqrt(-2.0 * log(u1)) * 0.70710678118654752;
    double sn, cs;
    sincospi(2.0 * u2, &sn, &cs);
    p[e] = make_double2(r * cs, r * sn);
  }
}

// aux_alpha = t^H ax for bordered stage-1 applies, and out[2..3] = t^H tr.
__global__ void __launch_bounds__(kRT) k_s1_trace(DevInst* __restrict__ st) {
  __shared__ double smem[32 * 4];
  DevInst& S = st[blockIdx.x];
  const double2* ax = (S.ax && S.aux_border) ? S.ax : nullptr;
  const double2* tr = S.tr;
  if (!ax && !tr) return;
  double acc[4] = {0, 0, 0, 0};
  for (int i = threadIdx.x; i < S.ndiag; i += blockDim.x) {
    const double w = S.sectors[S.diag_sector[i]].sqrt_f;
    const long long e = S.diag_index[i];
    if (ax) {
      acc[0] = fma(w, ax[e].x, acc[0]);
      acc[1] = fma(w, ax[e].y, acc[1]);
    }
    if (tr) {
      acc[2] = fma(w, tr[e].x, acc[2]);
      acc[3] = fma(w, tr[e].y, acc[3]);
    }
  }
  block_sum<4>(acc, smem);
  if (threadIdx.x == 0) {
    if (ax) S.aux_alpha = make_double2(acc[0], acc[1]);
    if (tr) {
      S.out[2] = acc[2];
      S.out[3] = acc[3];
    }
  }
}

constexpr int kBlockItems = kApplyThreads / 32;  // strip items that a block takes at once
constexpr int kRounds32 = 4;                     // times per entry of an FP32 apply list

// A warp's strip item of an instance with merged FP64 coefficients: y = scale
// L x + alpha v on the diagonal (reference coordinates), or y = L x when `plain`.
template <int V, bool NC>
__device__ __forceinline__ void strip_item(const DevInst& S, int item, const double2* x, double2* y, bool plain,
                                           double scale, const double2* alpha) {
  if (item >= S.p64.nitems) return;
  const StripItem it = S.p64.items[item];
  StripEntry<double, V, NC> E;
  if (!E.load(it, S.p64, threadIdx.x & 31)) return;
  double2 out = E.apply(x);
  if (plain) {  // block-uniform, its own exit: the scaling below must not be if-converted into it
    y[E.e] = out;
    return;
  }
  out.x *= scale;
  out.y *= scale;
  if (alpha != nullptr && E.diag) {
    const double v = S.sectors[it.sector].border_x;
    out.x = fma(alpha->x, v, out.x);
    out.y = fma(alpha->y, v, out.y);
  }
  y[E.e] = out;
}

template <bool NC>
__device__ __forceinline__ void strip_apply(const DevInst& S, int item, const double2* x, double2* y, double scale,
                                            const double2* alpha) {
  // an exact 1 is told by its bits: an FP64 comparison would go through the FP64 pipe
  const bool plain = alpha == nullptr && __double_as_longlong(scale) == 0x3ff0000000000000LL;
  switch (S.p64.variant) {
    case 0: return strip_item<0, NC>(S, item, x, y, plain, scale, alpha);
    case 1: return strip_item<1, NC>(S, item, x, y, plain, scale, alpha);
    case 2: return strip_item<2, NC>(S, item, x, y, plain, scale, alpha);
    case 3: return strip_item<3, NC>(S, item, x, y, plain, scale, alpha);
    case 4: return strip_item<4, NC>(S, item, x, y, plain, scale, alpha);
    case 5: return strip_item<5, NC>(S, item, x, y, plain, scale, alpha);
    default: return strip_item<6, NC>(S, item, x, y, plain, scale, alpha);
  }
}

// Strip items of an FP32 instance of a canonical plan: w = scale L x (+ alpha v on the diagonal)
// from the merged entry, row and column planes, one thread per entry.  The arithmetic of an
// entry is apply_tile_planes_to's (and sep_entries'), operation for operation, so every schedule
// gives the same bits.  Per entry: 32-48 bytes of planes and ten sources through L1, no window
// staging and no idle lanes.  What bounds it is the chain of loads behind an entry (work list,
// control block, record, then planes and sources), so a block takes four rounds of items per
// list entry.
template <bool PLUS, bool NC>
struct StripEntry32 {
  float4 c0, c1, c2, lv, rc;
  float2 xc, xu, xd, xl, xr, xo, v0, v1, w0, w1, xp, v2, w2;
  int e, m0, m2, sector;
  bool in, diag;

  __device__ __forceinline__ void load(const DevInst& S, const StripItem& it, const float2* x) {
    const int n = it.n;
    const int i = it.local0 + (threadIdx.x & 31);
    in = i < n * n;
    if (!in) return;
    constexpr int NE = PLUS ? 3 : 2;
    const int b = (int)((unsigned)i / (unsigned)n), a = i - b * n;
    e = it.off + i;
    sector = it.sector;
    diag = a == b;
    m0 = it.m0;
    m2 = it.m2;
    const float4* ep = S.planes.eplane + (long long)e * NE;
    c0 = __ldg(ep);
    c1 = __ldg(ep + 1);
    if (PLUS) c2 = __ldg(ep + 2);
    lv = __ldg(S.planes.lrow + it.loff + a);
    rc = __ldg(S.planes.rcol + it.loff + b);
    auto ld = [&](int k, bool ok) { return ok ? (NC ? __ldg(x + k) : x[k]) : make_float2(0.f, 0.f); };
    auto box = [](int u, int v, int m) { return (unsigned)u < (unsigned)m && (unsigned)v < (unsigned)m; };
    const int s0 = it.off0 + (a - 2) + (b - 2) * m0, g0 = it.off2 + a + b * m2;
    xc = ld(e, true);
    xu = ld(e - 1, a > 0);
    xd = ld(e + 1, a < n - 1);
    xl = ld(e - n, b > 0);
    xr = ld(e + n, b < n - 1);
    xo = ld(e - n - 1, a > 0 && b > 0);
    v0 = ld(s0, box(a - 2, b - 2, m0));
    v1 = ld(s0 + m0 + 1, box(a - 1, b - 1, m0));
    w0 = ld(g0, box(a, b, m2));
    w1 = ld(g0 + m2 + 1, box(a + 1, b + 1, m2));
    if (PLUS) {
      xp = ld(e + n + 1, a < n - 1 && b < n - 1);
      v2 = ld(s0 + 2 * (m0 + 1), box(a, b, m0));
      w2 = ld(g0 + 2 * (m2 + 1), box(a + 2, b + 2, m2));
    }
  }

  __device__ __forceinline__ void store(const DevInst& S, float2* y, const double2* alpha) const {
    if (!in) return;
    float2 acc = make_float2(0.f, 0.f);
    pmac(acc, c0.x, c0.y, xc);  // centre
    pmac(acc, lv.x, lv.y, xu);  // LEFT -1
    pmac(acc, lv.z, lv.w, xd);  // LEFT +1
    pmac(acc, rc.x, rc.y, xl);  // RIGHT -1
    pmac(acc, rc.z, rc.w, xr);  // RIGHT +1
    prmac(acc, c0.z, xo);       // own (-1,-1)
    if (m0 > 0) {
      prmac(acc, c0.w, v0);     // smaller (-2,-2)
      prmac(acc, c1.x, v1);     // smaller (-1,-1)
    }
    if (m2 > 0) {
      prmac(acc, c1.y, w0);     // larger (0,0)
      prmac(acc, c1.z, w1);     // larger (1,1)
    }
    if (PLUS) {
      prmac(acc, c1.w, xp);               // own (1,1)
      if (m0 > 0) prmac(acc, c2.x, v2);   // smaller (0,0)
      if (m2 > 0) prmac(acc, c2.y, w2);   // larger (2,2)
    }
    if (__double_as_longlong(S.scale) != 0x3ff0000000000000LL) {
      const float scale = (float)S.scale;
      acc.x *= scale;
      acc.y *= scale;
    }
    if (alpha != nullptr && diag) {
      const double2 al = *alpha;
      const double v = S.coords ? S.sectors[sector].border_z : S.sectors[sector].border_x;
      acc.x += (float)(al.x * v);
      acc.y += (float)(al.y * v);
    }
    y[e] = acc;
  }
};

// Items first, first + step, ... (at most `count`) by one warp; the record of the next item is
// in flight while an item is computed.
template <bool PLUS, bool NC>
__device__ __forceinline__ void strip_items32(const DevInst& S, int first, int step, int count, const float2* x,
                                              float2* y, const double2* alpha) {
  const int nitems = S.nitems32;
  if (first >= nitems) return;
  const StripItem* items = S.items32;
  StripItem next = items[first];
#pragma unroll 1
  for (int k = 0, item = first; k < count && item < nitems; ++k, item += step) {
    const StripItem it = next;
    if (k + 1 < count && item + step < nitems) next = items[item + step];
    StripEntry32<PLUS, NC> E;
    E.load(S, it, x);
    E.store(S, y, alpha);
  }
}

template <bool NC>
__device__ __forceinline__ void strip_apply32(const DevInst& S, int first, int step, int count, const float2* x,
                                              float2* y, const double2* alpha) {
  if (S.planes.plus)
    strip_items32<true, NC>(S, first, step, count, x, y, alpha);
  else
    strip_items32<false, NC>(S, first, step, count, x, y, alpha);
}

// Applies over the (instance, tile) list -- for an instance of a canonical plan an (instance,
// strip block) list.  AUX: ay = aux_scale L ax (+ border), FP64; otherwise the
// Arnoldi step w = scale L V_j (+ border) in the basis precision.
template <typename T, bool AUX>
__global__ void __launch_bounds__(kApplyThreads, sizeof(T) == 4 && !AUX ? 4 : 1)
    k_bapply(const DevInst* __restrict__ st, const int* __restrict__ tile_inst, const int* __restrict__ tile_local) {
  using T2 = typename Vec2<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T2* win = reinterpret_cast<T2*>(smem_raw);
  __shared__ int4 sterms[kMaxSectorTerms];
  __shared__ int ge[G_COUNT + 1];
  const DevInst& S = st[tile_inst[blockIdx.x]];
  if (AUX) {
    if (!S.ax) return;
    if (S.p64.items != nullptr) {  // block-uniform
      strip_apply<true>(S, tile_local[blockIdx.x] * kBlockItems + (threadIdx.x >> 5), S.ax, S.ay, S.aux_scale,
                        S.aux_border ? &S.aux_alpha : nullptr);
      return;
    }
    const DevTile tile = S.tiles[tile_local[blockIdx.x]];
    BorderArgs b{S.aux_scale, nullptr, 0};
    apply_tile<T>(S.sectors, S.terms, (const T2*)S.coef64, tile, (const T2*)S.ax, (T2*)S.ay, b,
                  S.aux_border ? &S.aux_alpha : nullptr, win, sterms, ge);
  } else {
    if (S.done) return;
    const T2* xin = (const T2*)S.V + (long long)S.j * S.ldv;
    if constexpr (sizeof(T) == sizeof(double)) {
      if (S.p64.items != nullptr) {  // block-uniform
        strip_apply<true>(S, tile_local[blockIdx.x] * kBlockItems + (threadIdx.x >> 5), xin, (double2*)S.w, S.scale, S.border ? &S.alpha : nullptr);
        return;
      }
    }
    if constexpr (sizeof(T) == sizeof(float)) {
      if (S.items32 != nullptr) {  // block-uniform
        strip_apply32<true>(S, tile_local[blockIdx.x] * kBlockItems * kRounds32 + (threadIdx.x >> 5), kBlockItems,
                            kRounds32, xin, (float2*)S.w, S.border ? &S.alpha : nullptr);
        return;
      }
    }
    const DevTile tile = S.tiles[tile_local[blockIdx.x]];
    BorderArgs b{S.scale, nullptr, S.coords};
    apply_tile<T>(S.sectors, S.terms, (const T2*)S.coefb, tile, xin, (T2*)S.w, b, S.border ? &S.alpha : nullptr, win,
                  sterms, ge);
  }
}

// Persistent FP32 Arnoldi-step apply w = scale L V_j (+ border) over the (instance, tile)
// list: gridDim.x blocks (a multiple of the SM count, picked by the engine's autotuner)
// stride over the list.  Tiles of instances with separable line planes run two-stage: a
// block computes one tile while the stage of its next such tile is in flight; any other
// tile runs the general stencil synchronously.  Per-entry arithmetic is k_bapply<float,
// false>'s, so w is bitwise the same for every grid size and for the one-block-per-tile
// launch.
__global__ void __launch_bounds__(kApplyThreads, 3)
    k_bapply_persist(const DevInst* __restrict__ st, const int* __restrict__ tile_inst,
                     const int* __restrict__ tile_local, int ntotal) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // work kind of list item i, block-uniform: 0 skip (instance stopped this cycle), 1 / 2
  // separable planes without / with the +1 diagonal shifts, 3 general stencil
  auto kind = [&](int i) -> int {
    if (i >= ntotal) return -1;
    const DevInst& S = st[tile_inst[i]];
    if (S.done) return 0;
    if (S.planes.srow != nullptr && S.coords == S.pwhich) return S.planes.plus ? 2 : 1;
    return 3;
  };
  auto issue = [&](int i, int k, int stage) {
    const DevInst& S = st[tile_inst[i]];
    const DevTile tile = S.tiles[tile_local[i]];
    const float2* xin = (const float2*)S.V + (long long)S.j * S.ldv;
    if (k == 2)
      sep_issue<kSepF4Plus>(S.sectors, tile, xin, S.planes, sep_stage(smem_raw, stage));
    else
      sep_issue<kSepF4>(S.sectors, tile, xin, S.planes, sep_stage(smem_raw, stage));
  };
  int i = blockIdx.x;
  int stage = 0;
  bool staged = false;  // item i's stage was issued by the previous iteration
  while (i < ntotal) {
    const int ki = kind(i);
    if (ki == 0) {
      i += gridDim.x;
      continue;
    }
    const DevInst& S = st[tile_inst[i]];
    const DevTile tile = S.tiles[tile_local[i]];
    const BorderArgs b{S.scale, nullptr, S.coords};
    const double2* al = S.border ? &S.alpha : nullptr;
    if (ki == 3) {  // nothing is in flight here: only separable tiles are prefetched
      float2* win = reinterpret_cast<float2*>(smem_raw);
      int4* sterms = reinterpret_cast<int4*>(smem_raw + 3 * kWinElems * sizeof(float2));
      int* ge = reinterpret_cast<int*>(sterms + kMaxSectorTerms);
      apply_tile<float>(S.sectors, S.terms, (const float2*)S.coefb, tile, (const float2*)S.V + (long long)S.j * S.ldv,
                        (float2*)S.w, b, al, win, sterms, ge);
      __syncthreads();  // the windows are restaged by the next item
      i += gridDim.x;
      continue;
    }
    if (!staged) issue(i, ki, stage);
    int j = i + gridDim.x;
    int kj = kind(j);
    while (kj == 0) {
      j += gridDim.x;
      kj = kind(j);
    }
    const bool pre = kj == 1 || kj == 2;
    if (pre) {
      issue(j, kj, stage ^ 1);
      cp_async_wait<1>();  // item i's group has landed, item j's stays in flight
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const StoreSink<float2> sink{(float2*)S.w};
    if (ki == 2)
      sep_compute<true>(S.sectors, tile, sink, b, al, sep_stage(smem_raw, stage));
    else
      sep_compute<false>(S.sectors, tile, sink, b, al, sep_stage(smem_raw, stage));
    __syncthreads();  // this stage is refilled by the prefetch of the item after j
    staged = pre;
    if (pre) stage ^= 1;
    i = kj < 0 ? ntotal : j;
  }
}

__global__ void __launch_bounds__(kRT) k_s1_resid(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst) {
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  double2* r = S.rout;
  if (!r) return;
  long long beg, end;
  chunk_range(S, blockIdx.x, beg, end);
  for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
    const double2 b = S.rb[e], a = S.ay[e];
    r[e] = make_double2(b.x - a.x, b.y - a.y);
  }
}

// |nrm0|^2 and |nrm1|^2 over one chunk; a combination's own norm is already there.
__global__ void __launch_bounds__(kRT)
    k_s1_norm_partial(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst, double* __restrict__ part) {
  __shared__ double2 red[kRT / 32];
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  const double2* a = S.nrm0 != S.cout ? S.nrm0 : nullptr;
  const double2* b = S.nrm1;
  if (!a && !b) return;
  long long beg, end;
  chunk_range(S, blockIdx.x, beg, end);
  double acc[2] = {0, 0};
  if (a)
    for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
      const double2 v = a[e];
      acc[0] = fma(v.y, v.y, fma(v.x, v.x, acc[0]));
    }
  if (b)
    for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
      const double2 v = b[e];
      acc[1] = fma(v.y, v.y, fma(v.x, v.x, acc[1]));
    }
  warp_transpose_sum<2>(acc);
  const int lane = threadIdx.x & 31;
  if (lane % 16 == 0) reinterpret_cast<double*>(&red[threadIdx.x >> 5])[lane / 16] = acc[0];
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0;
    for (int w = 0; w < kRT / 32; ++w) t += reinterpret_cast<const double*>(&red[w])[threadIdx.x];
    part[2 * blockIdx.x + threadIdx.x] = t;
  }
}

// Dots conj(ob_o) . obx of K observables over the thread's elements, summed over the warp.
template <int K>
__device__ __forceinline__ void obs_cols(const DevInst& S, long long beg, long long end, int o0, double* row) {
  double acc[2 * K];
#pragma unroll
  for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
  for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
    const double2 x = S.obx[e];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const double2 v = S.ob[(long long)(o0 + k) * S.dim + e];
      acc[2 * k] = fma(v.x, x.x, acc[2 * k]);
      acc[2 * k] = fma(v.y, x.y, acc[2 * k]);
      acc[2 * k + 1] = fma(v.x, x.y, acc[2 * k + 1]);
      acc[2 * k + 1] = fma(-v.y, x.x, acc[2 * k + 1]);
    }
  }
  warp_transpose_sum<2 * K>(acc);
  constexpr int span = 32 / (2 * K);
  const int lane = threadIdx.x & 31;
  if (lane % span == 0) row[2 * o0 + lane / span] = acc[0];
}

// Observable dots conj(ob_o) . obx over one chunk (FP64 data).
__global__ void __launch_bounds__(kRT)
    k_s1_obs_partial(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst, double2* __restrict__ partv) {
  __shared__ double red[kRT / 32][2 * kBatchMaxObs];
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  const int nob = S.nob;
  if (nob == 0) return;
  long long beg, end;
  chunk_range(S, blockIdx.x, beg, end);
  double* row = red[threadIdx.x >> 5];
  int o = 0;
  for (; o + 4 <= nob; o += 4) obs_cols<4>(S, beg, end, o, row);
  if (o + 2 <= nob) obs_cols<2>(S, beg, end, o, row), o += 2;
  if (o < nob) obs_cols<1>(S, beg, end, o, row);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * nob; i += blockDim.x) {
    double t = 0;
#pragma unroll
    for (int w = 0; w < kRT / 32; ++w) t += red[w][i];
    reinterpret_cast<double*>(partv + (long long)blockIdx.x * S.pstride)[i] = t;
  }
}

// Per-instance sums of chunk partials: one warp per value, fixed order.
__device__ __forceinline__ double2 warp_chunk_sum(const double2* partv, int begin, int nc, int stride, int i) {
  const int lane = threadIdx.x & 31;
  double sx = 0, sy = 0;
  for (int c = lane; c < nc; c += 32) {
    const double2 p = partv[(long long)(begin + c) * stride + i];
    sx += p.x;
    sy += p.y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    sx += __shfl_down_sync(0xffffffffu, sx, off);
    sy += __shfl_down_sync(0xffffffffu, sy, off);
  }
  return make_double2(sx, sy);
}

// A job's norms and observables from its chunk partials.
__global__ void __launch_bounds__(kRT)
    k_s1_final(const DevInst* __restrict__ st, const int* __restrict__ nchunks, const double* __restrict__ part,
               const double2* __restrict__ partv) {
  __shared__ double smem[32 * 2];
  const DevInst& S = st[blockIdx.x];
  const int warp = threadIdx.x >> 5, nc = nchunks[blockIdx.x];
  for (int o = warp; o < S.nob; o += blockDim.x >> 5) {
    const double2 v = warp_chunk_sum(partv, S.chunk_begin, nc, S.pstride, o);
    if ((threadIdx.x & 31) == 0) {
      S.out[4 + 2 * o] = v.x;
      S.out[5 + 2 * o] = v.y;
    }
  }
  if (!S.nrm0 && !S.nrm1) return;
  double acc[2] = {0, 0};
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    acc[0] += part[2 * (S.chunk_begin + c)];
    acc[1] += part[2 * (S.chunk_begin + c) + 1];
  }
  block_sum<2>(acc, smem, min((nc + 31) / 32, kRT / 32));
  if (threadIdx.x == 0) {
    S.out[0] = acc[0];
    S.out[1] = acc[1];
  }
}

// ---------------------------------------------------------------------------------------
// Arnoldi-step kernels
// ---------------------------------------------------------------------------------------

// V_0 = v0 / v0norm; the instance's first chunk also resets the GMRES right-hand side.
template <typename T2>
__global__ void __launch_bounds__(kRT) k_load_v0(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst) {
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  const double2* x = S.v0;
  if (!x) return;
  const double f = 1.0 / S.v0norm;
  long long beg, end;
  chunk_range(S, blockIdx.x, beg, end);
  T2* V = (T2*)S.V;
  for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
    const double2 v = x[e];
    st2(V + e, f * v.x, f * v.y);
  }
  if ((int)blockIdx.x == S.chunk_begin)
    for (int r = threadIdx.x; r < S.ldh; r += blockDim.x) S.g[r] = make_double2(r == 0 ? S.v0norm : 0.0, 0.0);
}

// The phases of one Arnoldi step are device functions of (job, input column j, chunk): the
// step kernels below launch one phase each, and k_cycle runs all phases of all steps of a
// small job set in one launch.  Pointers to data that the step writes carry no __restrict__
// and no read-only loads, as one kernel writes and reads them.

// t^H V_j for bordered cycles (whole block; every thread gets the value).
template <typename T2>
__device__ double2 step_trace(const DevInst& S, int j) {
  __shared__ double smem[32 * 2];
  __shared__ double2 total;
  const T2* x = (const T2*)S.V + (long long)j * S.ldv;
  double acc[2] = {0, 0};
  for (int i = threadIdx.x; i < S.ndiag; i += blockDim.x) {
    const double w = S.coords ? 1.0 : S.sectors[S.diag_sector[i]].sqrt_f;
    const double2 v = ld2(x + S.diag_index[i]);
    acc[0] = fma(w, v.x, acc[0]);
    acc[1] = fma(w, v.y, acc[1]);
  }
  block_sum<2>(acc, smem, min((S.ndiag + 31) / 32, kRT / 32));
  if (threadIdx.x == 0) total = make_double2(acc[0], acc[1]);
  __syncthreads();
  return total;
}

template <typename T2>
__global__ void __launch_bounds__(kRT) k_step_trace(DevInst* st) {
  DevInst& S = st[blockIdx.x];
  if (S.done || !S.border) return;
  const double2 a = step_trace<T2>(S, S.j);
  if (threadIdx.x == 0) S.alpha = a;
}

// ---- FP64-basis projections and updates ------------------------------------------------
// GB300's FP64 pipe bounds both (4 FMAs per element and basis vector against 16 bytes), so the
// reductions are kept off it as far as they go: a warp sums 2K values over its lanes by
// exchanging halves (2K - 1 additions, against 10K for K columns summed one by one), each lane
// holding 4 elements of w in registers across all columns.  N = 120, 31 columns: 43 us against 129 us
// (60 of them reductions) when every block summed eight columns one by one; 52 -> 4 us at one column.

// Projections of the lane's E elements onto K columns, summed over the warp into row[2 k ..].
template <int K, int E>
__device__ __forceinline__ void dot_cols64(const double2* V, long long ld, const double2 (&w)[4], int left,
                                           double* row) {
  double acc[2 * K];
#pragma unroll
  for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) v[q] = 32 * q < left ? V[k * ld + 32 * q] : make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < E; ++q) {
      acc[2 * k] = fma(v[q].x, w[q].x, acc[2 * k]);
      acc[2 * k] = fma(v[q].y, w[q].y, acc[2 * k]);
      acc[2 * k + 1] = fma(v[q].x, w[q].y, acc[2 * k + 1]);
      acc[2 * k + 1] = fma(-v[q].y, w[q].x, acc[2 * k + 1]);
    }
  }
  warp_transpose_sum<2 * K>(acc);
  constexpr int span = 32 / (2 * K);
  const int lane = threadIdx.x & 31;
  if (lane % span == 0) row[lane / span] = acc[0];
}

template <int E>
__device__ __forceinline__ void dot_range64(const double2* V, long long ld, const double2 (&w)[4], int left, int k,
                                            int k1, double* row) {
  for (; k + 16 <= k1; k += 16) dot_cols64<16, E>(V + k * ld, ld, w, left, row + 2 * k);
  if (k + 8 <= k1) dot_cols64<8, E>(V + k * ld, ld, w, left, row + 2 * k), k += 8;
  if (k + 4 <= k1) dot_cols64<4, E>(V + k * ld, ld, w, left, row + 2 * k), k += 4;
  if (k + 2 <= k1) dot_cols64<2, E>(V + k * ld, ld, w, left, row + 2 * k), k += 2;
  if (k < k1) dot_cols64<1, E>(V + k * ld, ld, w, left, row + 2 * k);
}

struct Dot64Smem {
  double row[8][2 * (kBatchMaxKrylov + 2)];  // per element group: (re, im) per column
  double norm[8];
};

// partv[c][i] = sum over chunk c of conj(V_i) w for i < nv, and ipart[c] = |w|^2 over the chunk
// (ipart != nullptr).  The chunk is cut into groups of 128 elements (4 per lane; chunks of 32
// and 64 elements: 1 and 2 per lane); the warps that a chunk of fewer than 8 groups leaves
// free take the groups' columns in parts.
__device__ __forceinline__ void step_dot64(const DevInst& S, int nv, int c, double2* partv, double* ipart,
                                           Dot64Smem& sm) {
  long long beg, end;
  chunk_range(S, c, beg, end);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = max(S.chunk / 128, 1), parts = 8 / groups;
  const int g = warp % groups, part = warp / groups;
  const long long e0 = beg + g * 128 + lane;
  const int left = (int)min(end - e0, 1024LL);  // element 32 q of the lane exists when 32 q < left
  double2 w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    w[q] = 32 * q < left ? ((const double2*)S.w)[e0 + 32 * q] : make_double2(0.0, 0.0);
  if (ipart != nullptr && part == 0) {
    double a = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (32 * q < S.chunk) a = fma(w[q].y, w[q].y, fma(w[q].x, w[q].x, a));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if (lane == 0) sm.norm[g] = a;
  }
  const int per = (nv + parts - 1) / parts;
  const int k = part * per, k1 = min(k + per, nv);
  const double2* V = (const double2*)S.V + e0;
  const long long ld = S.ldv;
  double* row = sm.row[g];
  if (S.chunk == 32)  // block-uniform
    dot_range64<1>(V, ld, w, left, k, k1, row);
  else if (S.chunk == 64)
    dot_range64<2>(V, ld, w, left, k, k1, row);
  else
    dot_range64<4>(V, ld, w, left, k, k1, row);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * nv; i += blockDim.x) {
    double t = sm.row[0][i];
    for (int q = 1; q < groups; ++q) t += sm.row[q][i];
    reinterpret_cast<double*>(partv + (long long)c * S.pstride)[i] = t;
  }
  if (ipart != nullptr && threadIdx.x == 0) {
    double t = sm.norm[0];
    for (int q = 1; q < groups; ++q) t += sm.norm[q];
    ipart[c] = t;
  }
  __syncthreads();  // sm is free for the block's next chunk
}

// The chunk kernels take an `again` word: null in the first pass (one block per chunk); in the
// second pass, which few jobs need, it says whether any does (k_step_norm), and a grid of a few
// blocks per SM returns at once or walks the chunks of the jobs that do.
template <typename F>
__device__ __forceinline__ void for_chunks(const DevInst* st, const int* chunk_inst, int nchunk, const int* again,
                                           const F& f) {
  if (again != nullptr && *again == 0) return;
  for (int c = blockIdx.x; c < nchunk; c += gridDim.x) {  // first pass: gridDim.x == nchunk
    const DevInst& S = st[chunk_inst[c]];
    if (!S.done && (again == nullptr || S.reorth)) f(S, c);
  }
}
constexpr int kSecondPassBlocks = 4 * 152;

__global__ void __launch_bounds__(kRT, 2)
    k_step_dot64(const DevInst* st, const int* chunk_inst, int nchunk, double2* partv, double* ipart,
                 const int* again) {
  __shared__ Dot64Smem sm;
  for_chunks(st, chunk_inst, nchunk, again,
             [&](const DevInst& S, int c) { step_dot64(S, S.j + 1, c, partv, ipart, sm); });
}

// which 0: hA, 1: hB (jobs that reorthogonalise).  Grid (instances, column groups): warp w of
// block (x, y) reduces column i = y * warps + w, so every column of every instance has its own
// warp (one warp walking several columns left a single SM reducing a long chunk list per
// column).
__global__ void __launch_bounds__(kRT)
    k_step_mdot_final(const DevInst* st, const int* __restrict__ nchunks, const double2* partv) {
  const DevInst& S = st[blockIdx.x];
  if (S.done || !S.reorth) return;
  const int i = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i > S.j) return;  // warp-uniform
  const double2 v = warp_chunk_sum(partv, S.chunk_begin, nchunks[blockIdx.x], S.pstride, i);
  if ((threadIdx.x & 31) == 0) S.hB[i] = v;
}

// Sums of a job's chunk partials (thread t sums partials t, t + 256, ..., then a deterministic
// block sum), to the whole block: x from a, y from b (b != nullptr).
__device__ __forceinline__ double2 job_norms(const DevInst& S, int nchunks, const double* a, const double* b) {
  __shared__ double smem[32 * 2];
  __shared__ double2 total;
  double acc[2] = {0, 0};
  for (int c = threadIdx.x; c < nchunks; c += blockDim.x) {
    acc[0] += a[S.chunk_begin + c];
    if (b != nullptr) acc[1] += b[S.chunk_begin + c];
  }
  block_sum<2>(acc, smem, min((nchunks + 31) / 32, kRT / 32));
  if (threadIdx.x == 0) total = make_double2(acc[0], acc[1]);
  __syncthreads();
  const double2 t = total;
  __syncthreads();  // total is free for the block's next job
  return t;
}

// The first-pass projections of a step into hA (grid as k_step_mdot_final's).
__global__ void __launch_bounds__(kRT)
    k_step_first_final(DevInst* st, const int* __restrict__ nchunks, const double2* partv) {
  DevInst& S = st[blockIdx.x];
  if (S.done) return;
  const int i = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i > S.j) return;  // warp-uniform
  const double2 v = warp_chunk_sum(partv, S.chunk_begin, nchunks[blockIdx.x], S.pstride, i);
  if ((threadIdx.x & 31) == 0) S.hA[i] = v;
}

// 1 / |w| (zero on an exact breakdown).
__device__ __forceinline__ double inverse_norm(double rem2) {
  const double r = sqrt(rem2);
  return r > 0 ? 1.0 / r : 0.0;
}

// The same for the whole block: one warp computes it, as the FP64 root and quotient of eight
// warps would queue on the pipe.
__device__ __forceinline__ double block_inverse_norm(double rem2) {
  __shared__ double inv;
  __syncthreads();  // an earlier value has been read
  if (threadIdx.x < 32) {
    const double f = inverse_norm(rem2);
    if (threadIdx.x == 0) inv = f;
  }
  __syncthreads();
  return inv;
}

// After the first update (whole block): |L V_j|^2, |w1|^2 and whether the job reorthogonalises.
// Selective reorthogonalisation (Daniel, Gragg, Kaufman, Stewart, Math. Comp. 30, 772 (1976)):
// when |w1|^2 >= |w0|^2 / 2 (w0 = L V_j before any projection) the first pass has left w
// orthogonal to the basis to working precision, and the second pass is skipped (zero hB).
// `store`: this block writes the job's record.
struct StepNorms {
  double rem2;
  bool reorth;
};
__device__ __forceinline__ StepNorms step_norm1(DevInst& S, int nv, int nchunks, const double* part,
                                                const double* part1, bool store) {
  const double2 v = job_norms(S, nchunks, part, part1);
  const bool reorth = v.y < 0.5 * v.x;
  if (store) {
    if (threadIdx.x == 0) {
      S.image2 = v.x;
      S.rem2 = v.y;
      S.reorth = reorth ? 1 : 0;
      if (!reorth) S.inv = inverse_norm(v.y);
    }
    for (int i = threadIdx.x; i < nv; i += blockDim.x) S.hB[i] = make_double2(0.0, 0.0);
  }
  return StepNorms{v.y, reorth};
}

// One block per job.  second 0: step_norm1; 1: |w|^2 after the second update of a job that
// reorthogonalised.
__global__ void __launch_bounds__(kRT)
    k_step_norm(DevInst* st, const int* __restrict__ nchunks, const double* part, const double* part1, int second,
                int* again) {
  DevInst& S = st[blockIdx.x];
  if (S.done) return;
  if (!second) {
    const StepNorms r = step_norm1(S, S.j + 1, nchunks[blockIdx.x], part, part1, true);
    if (r.reorth && threadIdx.x == 0) atomicExch(again, 1);
  } else if (S.reorth) {
    const double2 v = job_norms(S, nchunks[blockIdx.x], part, nullptr);
    if (threadIdx.x == 0) {
      S.rem2 = v.x;
      S.inv = inverse_norm(v.x);
    }
  }
}

// w -= sum_i V_i h_i over chunk c and part[c] = |w|^2 of the result.  A thread holds up to 4
// elements; chunks of fewer than 256 elements split the columns between parts of the block.
struct Axpy64Smem {
  double2 h[kBatchMaxKrylov + 2];
  double2 share[kRT];
  double red[32];
};

__device__ __forceinline__ void axpy_cols64(const double2* V, long long ld, const double2* h, int k0, int k1,
                                            double2& w) {
#pragma unroll 8
  for (int i = k0; i < k1; ++i) {
    const double2 v = V[i * ld];
    const double2 c = h[i];
    w.x = fma(-v.x, c.x, w.x);
    w.x = fma(v.y, c.y, w.x);
    w.y = fma(-v.x, c.y, w.y);
    w.y = fma(-v.y, c.x, w.y);
  }
}

// sm.h holds the projections (the caller has synchronised).
__device__ __forceinline__ void step_axpy64(const DevInst& S, int nv, int c, double* part, Axpy64Smem& sm) {
  long long beg, end;
  chunk_range(S, c, beg, end);
  const double2* V = (const double2*)S.V;
  double2* w = (double2*)S.w;
  const long long ld = S.ldv;
  double acc[1] = {0};
  if (S.chunk < kRT) {  // block-uniform
    const int at = threadIdx.x % S.chunk, p = threadIdx.x / S.chunk, parts = kRT / S.chunk;
    const long long e = beg + at;
    const int per = (nv + parts - 1) / parts;
    double2 v = make_double2(0.0, 0.0);
    if (e < end) {
      if (p == 0) v = w[e];
      axpy_cols64(V + e, ld, sm.h, p * per, min(p * per + per, nv), v);
    }
    sm.share[threadIdx.x] = v;
    __syncthreads();
    if (p == 0 && e < end) {
      for (int q = 1; q < parts; ++q) {
        v.x += sm.share[q * S.chunk + at].x;
        v.y += sm.share[q * S.chunk + at].y;
      }
      w[e] = v;
      acc[0] = fma(v.y, v.y, v.x * v.x);
    }
  } else {
    for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
      double2 v = w[e];
      axpy_cols64(V + e, ld, sm.h, 0, nv, v);
      w[e] = v;
      acc[0] = fma(v.x, v.x, acc[0]);
      acc[0] = fma(v.y, v.y, acc[0]);
    }
  }
  block_sum<1>(acc, sm.red, min(S.chunk, kRT) / 32);
  if (threadIdx.x == 0) part[c] = acc[0];
  __syncthreads();  // sm is free for the block's next chunk
}

__global__ void __launch_bounds__(kRT, 2)
    k_step_axpy64(const DevInst* st, const int* chunk_inst, int nchunk, double* part, const int* again) {
  __shared__ Axpy64Smem sm;
  for_chunks(st, chunk_inst, nchunk, again, [&](const DevInst& S, int c) {
    const double2* h = again ? S.hB : S.hA;
    for (int i = threadIdx.x; i <= S.j; i += blockDim.x) sm.h[i] = h[i];
    __syncthreads();
    step_axpy64(S, S.j + 1, c, part, sm);
  });
}

// V_{j+1} = f w over chunk c, f = 1 / |w|.
__device__ __forceinline__ void step_normalize64(const DevInst& S, int j, int c, double f) {
  long long beg, end;
  chunk_range(S, c, beg, end);
  const double2* w = (const double2*)S.w;
  double2* out = (double2*)S.V + (long long)(j + 1) * S.ldv;
  for (long long e = beg + threadIdx.x; e < end; e += blockDim.x) {
    const double2 v = w[e];
    out[e] = make_double2(f * v.x, f * v.y);
  }
}

__global__ void __launch_bounds__(kRT) k_step_normalize64(const DevInst* st, const int* chunk_inst) {
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  if (S.done) return;
  step_normalize64(S, S.j, blockIdx.x, S.inv);
}

// ---- FP32-basis CGS2 kernels: pairs of complex elements per 16-byte load ---------------
// Basis columns and the image vector have an even, zero-padded stride, so element pairs
// never straddle a column; padding entries stay zero through every update.

__device__ __forceinline__ void pair_range(const DevInst& S, int c, long long& beg, long long& end) {
  beg = (long long)(c - S.chunk_begin) * (S.chunk / 2);
  end = min(beg + (long long)(S.chunk / 2), (S.dim + 1) / 2);
}

// Warp sum of double-float values in FP32 arithmetic (GB300's FP64 pipe is narrow: the
// per-column reductions stay off it); the result is valid in lane 0.
__device__ __forceinline__ DF warp_df_sum(DF v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const DF o{__shfl_down_sync(0xffffffffu, v.hi, off), __shfl_down_sync(0xffffffffu, v.lo, off)};
    v = df_sum(v, o);
  }
  return v;
}

// Block sum of one double-float value; the FP64 result is valid in thread 0.
__device__ __forceinline__ double block_df_sum(DF v, float2* smem) {
  v = warp_df_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) smem[warp] = make_float2(v.hi, v.lo);
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    DF t{0.f, 0.f};
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t = df_sum(t, DF{smem[i].x, smem[i].y});
    r = (double)t.hi + (double)t.lo;
  }
  return r;
}

// CGS2 projections for an FP32 basis: partv[c][i] = conj(V_i) . w over chunk c for every
// i <= j.  The block stages its chunk of w (CH elements) in shared memory and streams every
// basis column once: per column it forms each pair term (two complex products) in FP32 and
// accumulates the terms in double-float (no rounding error in the accumulation), then the
// warp sums its lanes in FP64 into shared memory.

__device__ __forceinline__ void pair_terms(const float4 a, const float4 b, DF& re, DF& im) {
  df_add(re, fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))));
  df_add(im, fmaf(a.x, b.y, fmaf(-a.y, b.x, fmaf(a.z, b.w, -(a.w * b.z)))));
}

// With ipart (first pass of a step) the block also writes the double-float |w|^2 partial of
// its chunk for the image norm |L V_j| (the expv error estimate and the reorthogonalisation
// test) -- the same pairs in the same order as a separate sweep over w would take -- while w
// is staged anyway.
//
// The lane sums of K columns exchange halves of the accumulators (2K - 1 double-float additions
// and as many shuffles, against 10K one value at a time, which at 1024 elements per chunk were
// two thirds of the instructions); each value is still summed over the same tree of lanes.
template <int CH>
struct Dot32Smem {
  float4 w[CH / 2];
  // per warp: double-float (hi, lo) of re and im of each basis column (at most kBatchMaxKrylov
  // + 1); sized to the engine's Krylov limit so the block stays inside 48 KB of shared memory
  float2 red[kRT / 32][2 * (kBatchMaxKrylov + 2)];
};

// K columns from V4 on: row[2 k], row[2 k + 1] = the warp's sums.
template <int K, int CH>
__device__ __forceinline__ void dot_cols32(const float4* V4, long long ld4, const float4* w, int npair, float2* row) {
  constexpr int kPairs = CH / 2 / kRT;  // element pairs per thread and chunk
  constexpr int kStep = K * kPairs <= 16 ? kPairs : 2;  // pairs whose K loads are in flight together
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  DF acc[2 * K];
#pragma unroll
  for (int k = 0; k < 2 * K; ++k) acc[k] = DF{0.f, 0.f};
#pragma unroll 1
  for (int q0 = 0; q0 < kPairs; q0 += kStep) {
    float4 v[K][kStep];
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int q = 0; q < kStep; ++q) {
        const int p = threadIdx.x + (q0 + q) * kRT;
        v[k][q] = p < npair ? V4[k * ld4 + p] : zero;
      }
#pragma unroll
    for (int q = 0; q < kStep; ++q) {
      const float4 wv = w[threadIdx.x + (q0 + q) * kRT];
#pragma unroll
      for (int k = 0; k < K; ++k) pair_terms(v[k][q], wv, acc[2 * k], acc[2 * k + 1]);
    }
  }
  warp_transpose_sum<2 * K>(acc);
  constexpr int span = 32 / (2 * K);
  const int lane = threadIdx.x & 31;
  if (lane % span == 0) row[lane / span] = make_float2(acc[0].hi, acc[0].lo);
}

// KMAX: columns per group, by the registers that the kernel has (every split sums alike).
template <int CH, int KMAX>
__device__ __forceinline__ void step_dot32(const DevInst& S, int nv, int c, double2* partv, double* ipart,
                                           Dot32Smem<CH>& sm) {
  constexpr int kPairs = CH / 2 / kRT;
  long long beg, end;
  pair_range(S, c, beg, end);
  const int npair = (int)(end - beg);
  const float4* w4 = reinterpret_cast<const float4*>(S.w) + beg;
  const float4* V4 = reinterpret_cast<const float4*>(S.V) + beg;
  const long long ld4 = S.ldv / 2;
  DF nrm{0.f, 0.f};
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    const int p = threadIdx.x + q * kRT;
    const float4 wv = p < npair ? w4[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    sm.w[p] = wv;
    if (p < npair) df_add(nrm, fmaf(wv.x, wv.x, fmaf(wv.y, wv.y, fmaf(wv.z, wv.z, wv.w * wv.w))));
  }
  if (ipart != nullptr) {  // block-uniform
    const double r = block_df_sum(nrm, &sm.red[0][0]);
    if (threadIdx.x == 0) ipart[c] = r;
    __syncthreads();  // red is free
  }
  // a thread reads back its own entries of sm.w only
  float2* row = sm.red[threadIdx.x >> 5];
  int k = 0;
  for (; k + KMAX <= nv; k += KMAX) dot_cols32<KMAX, CH>(V4 + k * ld4, ld4, sm.w, npair, row + 2 * k);
  if (KMAX > 4 && k + 4 <= nv) dot_cols32<4, CH>(V4 + k * ld4, ld4, sm.w, npair, row + 2 * k), k += 4;
  if (k + 2 <= nv) dot_cols32<2, CH>(V4 + k * ld4, ld4, sm.w, npair, row + 2 * k), k += 2;
  if (k < nv) dot_cols32<1, CH>(V4 + k * ld4, ld4, sm.w, npair, row + 2 * k);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * nv; i += blockDim.x) {
    DF t{0.f, 0.f};
#pragma unroll
    for (int wdx = 0; wdx < kRT / 32; ++wdx) t = df_sum(t, DF{sm.red[wdx][i].x, sm.red[wdx][i].y});
    reinterpret_cast<double*>(partv + (long long)c * S.pstride)[i] = (double)t.hi + (double)t.lo;
  }
  __syncthreads();  // sm is free for the block's next chunk
}

template <int CH>
__global__ void __launch_bounds__(kRT, 3)
    k_step_mdot_f32(const DevInst* st, const int* chunk_inst, int nchunk, double2* partv, double* ipart,
                    const int* again) {
  __shared__ Dot32Smem<CH> sm;
  for_chunks(st, chunk_inst, nchunk, again,
             [&](const DevInst& S, int c) { step_dot32<CH, 4>(S, S.j + 1, c, partv, ipart, sm); });
}

// cout (+)= sum_k ccoef[k] V_k for an FP32 basis in double-float arithmetic: each FP64
// coefficient is split into hi + lo floats, hi * v is formed exactly (FMA residual), lo * v
// in FP32, and the sum is carried as a double-float per component, so the FP64 output
// matches an FP64 accumulation to ~1e-14 while the FP64 pipe stays idle.
__global__ void __launch_bounds__(kRT)
    k_s1_combine_f32(const DevInst* __restrict__ st, const int* __restrict__ chunk_inst, double* __restrict__ part) {
  __shared__ float4 cs[kBatchMaxKrylov + 2];  // (re.hi, re.lo, im.hi, im.lo)
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  double2* out = S.cout;
  if (!out) return;
  const int nc = S.ccount;
  for (int i = threadIdx.x; i < nc; i += blockDim.x) {
    const double2 c = S.ccoef[i];
    const float rh = (float)c.x, ih = (float)c.y;
    cs[i] = make_float4(rh, (float)(c.x - (double)rh), ih, (float)(c.y - (double)ih));
  }
  __syncthreads();
  long long beg, end;
  pair_range(S, blockIdx.x, beg, end);
  const float4* __restrict__ V4 = reinterpret_cast<const float4*>(S.V);
  const long long ld4 = S.ldv / 2;
  const int acc = S.cacc;
  double nrm = 0;
  for (long long p = beg + threadIdx.x; p < end; p += blockDim.x) {
    DF y0r{0.f, 0.f}, y0i{0.f, 0.f}, y1r{0.f, 0.f}, y1i{0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < nc; ++k) {
      const float4 v = V4[(long long)k * ld4 + p];
      const float4 c = cs[k];
      df_axpy(y0r, c.x, c.y, v.x);
      df_axpy(y0r, -c.z, -c.w, v.y);
      df_axpy(y0i, c.x, c.y, v.y);
      df_axpy(y0i, c.z, c.w, v.x);
      df_axpy(y1r, c.x, c.y, v.z);
      df_axpy(y1r, -c.z, -c.w, v.w);
      df_axpy(y1i, c.x, c.y, v.w);
      df_axpy(y1i, c.z, c.w, v.z);
    }
    auto put = [&](long long e, DF r, DF i) {
      double ox = (double)r.hi + (double)r.lo, oy = (double)i.hi + (double)i.lo;
      if (acc) {
        const double2 o = out[e];
        ox += o.x;
        oy += o.y;
      }
      out[e] = make_double2(ox, oy);
      nrm = fma(oy, oy, fma(ox, ox, nrm));
    };
    put(2 * p, y0r, y0i);
    if (2 * p + 1 < S.dim) put(2 * p + 1, y1r, y1i);
  }
  combined_norm(S, nrm, part);
}

// w -= sum_i V_i h_i over chunk c of an FP32 basis, FP32 update, and the double-float |w|^2
// partial of the result.
struct Axpy32Smem {
  float2 h[kBatchMaxKrylov + 2];
  float2 red[32];
};

// sm.h holds the projections (the caller has synchronised).
__device__ __forceinline__ void step_axpy32(const DevInst& S, int nv, int c, double* part, Axpy32Smem& sm) {
  long long beg, end;
  pair_range(S, c, beg, end);
  float4* w4 = reinterpret_cast<float4*>(S.w);
  const float4* V4 = reinterpret_cast<const float4*>(S.V);
  const long long ld4 = S.ldv / 2;
  DF nrm{0.f, 0.f};
  for (long long p = beg + threadIdx.x; p < end; p += blockDim.x) {
    float4 wv = w4[p];
#pragma unroll 8
    for (int i = 0; i < nv; ++i) {
      const float4 v = V4[(long long)i * ld4 + p];
      const float2 cf = sm.h[i];
      wv.x = fmaf(-v.x, cf.x, wv.x);
      wv.x = fmaf(v.y, cf.y, wv.x);
      wv.y = fmaf(-v.x, cf.y, wv.y);
      wv.y = fmaf(-v.y, cf.x, wv.y);
      wv.z = fmaf(-v.z, cf.x, wv.z);
      wv.z = fmaf(v.w, cf.y, wv.z);
      wv.w = fmaf(-v.z, cf.y, wv.w);
      wv.w = fmaf(-v.w, cf.x, wv.w);
    }
    w4[p] = wv;
    df_add(nrm, fmaf(wv.x, wv.x, fmaf(wv.y, wv.y, fmaf(wv.z, wv.z, wv.w * wv.w))));
  }
  const double r = block_df_sum(nrm, sm.red);
  if (threadIdx.x == 0) part[c] = r;
  __syncthreads();  // sm is free for the block's next chunk
}

__global__ void __launch_bounds__(kRT)
    k_step_maxpy_f32(const DevInst* st, const int* chunk_inst, int nchunk, double* part, const int* again) {
  __shared__ Axpy32Smem sm;
  for_chunks(st, chunk_inst, nchunk, again, [&](const DevInst& S, int c) {
    const double2* h = again ? S.hB : S.hA;
    for (int i = threadIdx.x; i <= S.j; i += blockDim.x) sm.h[i] = make_float2((float)h[i].x, (float)h[i].y);
    __syncthreads();
    step_axpy32(S, S.j + 1, c, part, sm);
  });
}

// V_{j+1} = f w over chunk c, f = 1 / |w|, FP32 basis.
__device__ __forceinline__ void step_normalize32(const DevInst& S, int j, int c, float f) {
  long long beg, end;
  pair_range(S, c, beg, end);
  const float4* w4 = reinterpret_cast<const float4*>(S.w);
  float4* out = reinterpret_cast<float4*>(S.V) + (long long)(j + 1) * (S.ldv / 2);
  for (long long p = beg + threadIdx.x; p < end; p += blockDim.x) {
    const float4 v = w4[p];
    out[p] = make_float4(f * v.x, f * v.y, f * v.z, f * v.w);
  }
}

__global__ void __launch_bounds__(kRT) k_step_normalize_f32(const DevInst* st, const int* chunk_inst) {
  const DevInst& S = st[chunk_inst[blockIdx.x]];
  if (S.done) return;
  step_normalize32(S, S.j, blockIdx.x, (float)S.inv);
}

// Per instance (one warp): records Hessenberg column j, applies the GMRES rotations and stop
// test (krylov.jl:759-777).  True (in every lane) when the job takes no further step.  An FP64
// instruction of one lane holds the pipe as long as one of 32, so the work is spread over the
// lanes: the rotations of the column are a linear recurrence in the running entry t (t' = c h -
// conj(s) t) whose products with c h are formed for all rows at once and whose real and
// imaginary part advance in two lanes together; the rotated entries c t + s h follow for all
// rows at once.  25 rotations: 25 -> 10 us against one lane doing the whole column.  Not inlined:
// the step kernel and k_cycle share one body, so both round alike.
struct FinishSmem {
  double2 h[kBatchMaxKrylov + 2];   // the new column
  double2 t[kBatchMaxKrylov + 2];   // running entry before rotation r
  double2 ch[kBatchMaxKrylov + 2];  // c_r h_{r+1}
  double2 sn[kBatchMaxKrylov + 2];
  double cs[kBatchMaxKrylov + 2];
};

__device__ __noinline__ bool step_finish(DevInst& S, int j, FinishSmem& sm) {
  const int lane = threadIdx.x & 31;
  const int ld = S.ldh;
  double2* col = S.H + (long long)j * ld;
  double2* cs = S.csn;
  double2* sn = S.csn + ld;
  const double root = sqrt(lane & 1 ? S.image2 : S.rem2);
  const double rem = __shfl_sync(0xffffffffu, root, 0);
  if (lane == 1) S.image[j] = root;
  if (lane == 0) S.kdone = j + 1;
  for (int r = lane; r < ld; r += 32)
    sm.h[r] = r <= j       ? make_double2(S.hA[r].x + S.hB[r].x, S.hA[r].y + S.hB[r].y)
              : r == j + 1 ? make_double2(rem, 0.0)
                           : make_double2(0.0, 0.0);
  bool stop = (j + 1 >= S.m) || rem == 0.0 || (long long)(j + 1) == S.dim;
  __syncwarp();
  if (S.givens) {
    for (int r = lane; r < j; r += 32) {
      const double c = cs[r].x;
      sm.cs[r] = c;
      sm.sn[r] = sn[r];
      sm.ch[r] = make_double2(c * sm.h[r + 1].x, c * sm.h[r + 1].y);
    }
    __syncwarp();
    // even lanes carry Re t, odd lanes Im t
    const int im = lane & 1;
    double mine = im ? sm.h[0].y : sm.h[0].x;
#pragma unroll 4
    for (int r = 0; r < j; ++r) {
      const double other = __shfl_xor_sync(0xffffffffu, mine, 1);
      if (lane < 2) reinterpret_cast<double*>(sm.t)[2 * r + im] = mine;
      const double2 s = sm.sn[r], ch = sm.ch[r];
      // -conj(s) t: Re = -(s.x t.x + s.y t.y), Im = -(s.x t.y - s.y t.x)
      mine = fma(-s.x, mine, fma(im ? s.y : -s.y, other, im ? ch.y : ch.x));
    }
    const double other = __shfl_xor_sync(0xffffffffu, mine, 1);
    const double2 a = im ? make_double2(other, mine) : make_double2(mine, other);  // entry j, rotated
    __syncwarp();
    for (int base = 0; base < j; base += 32) {
      const int r = base + lane;
      double2 v = make_double2(0.0, 0.0);
      if (r < j) {
        const double2 t = sm.t[r], h = sm.h[r + 1], s = sm.sn[r];
        const double c = sm.cs[r];
        v = make_double2(fma(c, t.x, fma(s.x, h.x, -s.y * h.y)), fma(c, t.y, fma(s.x, h.y, s.y * h.x)));
      }
      __syncwarp();  // h[r] is the next lane's h_{r+1}
      if (r < j) sm.h[r] = v;
      __syncwarp();
    }
    // complex Givens rotation of (a, rem) (krylov.jl:710-716; rem is real and not negative):
    // c = |a| / |(a, rem)|, s = (a / |a|) rem / |(a, rem)|, the four quotients in four lanes
    double c;
    double2 s;
    if (rem == 0.0) {
      c = 1.0;
      s = make_double2(0.0, 0.0);
    } else if (a.x == 0.0 && a.y == 0.0) {
      c = 0.0;
      s = make_double2(1.0, 0.0);
    } else {
      // |a| and |(a, rem)|; their squares are formed unless they could leave the FP64 range
      const double big = fmax(fabs(a.x), fabs(a.y));
      double aa, nn;
      if (big > 1e-140 && fmax(big, rem) < 1e140) {
        const double a2 = fma(a.x, a.x, a.y * a.y);
        const double two = sqrt(lane & 1 ? fma(rem, rem, a2) : a2);
        aa = __shfl_sync(0xffffffffu, two, 0);
        nn = __shfl_sync(0xffffffffu, two, 1);
      } else {
        aa = hypot(a.x, a.y);
        nn = hypot(aa, rem);
      }
      const int q = lane & 3;
      const double quot = (q == 0 ? aa : q == 1 ? rem : q == 2 ? a.x : a.y) / (q < 2 ? nn : aa);
      c = __shfl_sync(0xffffffffu, quot, 0);
      const double f = __shfl_sync(0xffffffffu, quot, 1);
      s = make_double2(f * __shfl_sync(0xffffffffu, quot, 2), f * __shfl_sync(0xffffffffu, quot, 3));
    }
    const double2 g1 = S.g[j], g2 = S.g[j + 1];
    const double2 sg2 = cmul(s, g2), csg1 = cmul(conjd(s), g1);
    const double2 n1 = make_double2(fma(c, g1.x, sg2.x), fma(c, g1.y, sg2.y));
    const double2 n2 = make_double2(fma(c, g2.x, -csg1.x), fma(c, g2.y, -csg1.y));
    __syncwarp();
    if (lane == 0) {
      cs[j] = make_double2(c, 0.0);
      sn[j] = s;
      sm.h[j] = make_double2(fma(c, a.x, s.x * rem), fma(c, a.y, s.y * rem));
      sm.h[j + 1] = make_double2(0.0, 0.0);
      S.g[j] = n1;
      S.g[j + 1] = n2;
    }
    const double tol = S.tol;
    if (tol > 1e-140 ? fma(n2.x, n2.x, n2.y * n2.y) <= tol * tol : hypot(n2.x, n2.y) <= tol) stop = true;
  }
  __syncwarp();
  for (int r = lane; r < ld; r += 32) col[r] = sm.h[r];
  __syncwarp();
  return stop;
}

__global__ void __launch_bounds__(32) k_step_finish(DevInst* st, int* again) {
  __shared__ FinishSmem sm;
  DevInst& S = st[blockIdx.x];
  if (blockIdx.x == 0 && threadIdx.x == 0) *again = 0;  // for the next step
  if (S.done) return;
  const int j = S.j;
  const bool stop = step_finish(S, j, sm);
  if (threadIdx.x == 0) {
    if (stop)
      S.done = 1;
    else
      S.j = j + 1;
  }
}

// ---- one launch per Krylov cycle -------------------------------------------------------
// The m steps of a small job set in one cooperative launch: its blocks walk each phase's work
// list and meet at a grid barrier between phases.  As separate launches (one graph of 11 nodes
// per step) the phases of such sets last about as long as a launch takes to start and drain.
// Per entry, chunk and job the arithmetic is that of the step kernels.  Measured per Arnoldi
// step, graph -> one launch: N = 8 FP64 68 -> 24 us, N = 16 GMRES(50) about 120 -> 30 us, N = 120
// FP32 63 -> 27 us (m = 30).  A barrier takes about 1 us and a phase of a small set 3-7 us, most
// of it the latency of loads that miss L1 (the barrier's fence empties it) and of FP64
// instructions (64 cycles each per quarter of an SM).

// Grid barrier: arrivals are counted up over the whole launch.  A block that waits in vain
// raises err, which ends every wait of the launch; the host reads it after the cycle.  Without one
// (bar null) the grid is one cluster and the barrier is the cluster's, in hardware: an interval
// of N = 8 (seven blocks, 30 steps) takes 0.87 -> 0.73 ms.  Every block leaves the cycle at the
// same barrier, and a cluster barrier waits for threads that have not exited only.
struct GridBar {
  unsigned count;
  int err;
};
constexpr int kGridWaitLimit = 1 << 24;  // polls, several seconds

// Arrival of this block; its writes so far are visible to blocks that wait for it.
__device__ __forceinline__ void grid_arrive(GridBar* bar, unsigned& target) {
  if (bar != nullptr) __syncthreads();
  target += gridDim.x;
  if (bar == nullptr) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    return;
  }
  if (gridDim.x > 1 && threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&bar->count, 1u);
  }
}

// Waits for the arrival of every block; false when the launch has given up.
__device__ __forceinline__ bool grid_wait(GridBar* bar, unsigned target) {
  if (bar == nullptr) {
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
  if (gridDim.x == 1) return true;
  __shared__ int ok;
  if (threadIdx.x == 0) {
    ok = 1;
    for (int it = 0;; ++it) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&bar->count) : "memory");
      if ((int)(seen - target) >= 0) break;
      if (it >= kGridWaitLimit || ((it & 1023) == 1023 && atomicAdd(&bar->err, 0) != 0)) {
        atomicExch(&bar->err, 1);
        ok = 0;
        break;
      }
    }
    __threadfence();  // the other blocks' writes after it
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ bool grid_sync(GridBar* bar, unsigned& target) {
  grid_arrive(bar, target);
  return grid_wait(bar, target);
}

// Sum of a job's nc <= 32 chunk partials of projection i in the order of warp_chunk_sum (lane c
// holds partial c, halves added pairwise), by one thread.
__device__ __noinline__ double few_chunk_sum(const double2* partv, int begin, int nc, int stride, int value) {
  const double* p = reinterpret_cast<const double*>(partv) + (long long)begin * stride * 2 + value;
  double v[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) v[c] = c < nc ? p[(long long)c * stride * 2] : 0.0;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int c = 0; c < off; ++c)
      if (c + off < nc) v[c] += v[c + off];  // uniform; adding the zero of a missing chunk changes nothing
  return v[0];
}
constexpr int kFewChunks = 32;

template <bool F32>
__global__ void __launch_bounds__(kRT, 2)
    k_cycle(DevInst* st, int n, const int* chunk_inst, int nchunk, const int* item_inst, const int* item_local,
            int nitem, const int* nchunks, double2* partv, double* part, int steps, int border, GridBar* bar) {
  __shared__ __align__(16) union {
    Dot64Smem dot64;
    Axpy64Smem axpy64;
    Dot32Smem<kBatchChunkSmall> dot32;
    Axpy32Smem axpy32;
    FinishSmem finish;
  } sm;
  __shared__ double2 tr;
  // a single job's control block, for the fields that stay as they are
  __shared__ __align__(16) unsigned char fixed_raw[sizeof(DevInst)];
  DevInst& fixed = *reinterpret_cast<DevInst*>(fixed_raw);
  using T2 = typename Vec2<typename std::conditional<F32, float, double>::type>::type;
  const int nblk = gridDim.x, blk = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned target = 0;  // arrivals at the barrier that comes next
  double* part1 = part + nchunk;
  // A single job: its norms and its trace are reduced by every block for itself, which costs
  // less than a designated block and a barrier.
  const bool one = n == 1;
  // Its last block takes no share of the applies and, the grid having a block more than there
  // are chunks, of the chunk phases of smaller jobs: it arrives at the apply's barrier before it
  // starts the finish, so that only the end of the projections waits for it.
  const int workers = one && nblk > 1 ? nblk - 1 : nblk;
  for (int i = threadIdx.x; one && i < (int)(sizeof(DevInst) / 4); i += kRT)
    reinterpret_cast<int*>(&fixed)[i] = reinterpret_cast<const int*>(st)[i];
  __syncthreads();
  auto job = [&](int i) -> const DevInst& { return one ? fixed : st[i]; };
  const bool own_trace = one && border && st[0].border && st[0].ndiag <= 4 * kRT;
  const int nc0 = nchunks[0];
  bool many = false;  // some job's projections are reduced in a phase of their own
  for (int i = threadIdx.x; i < n; i += kRT) many = many || nchunks[i] > kFewChunks;
  many = __syncthreads_or(many);
  for (int j = 0;; ++j) {
    // The finish of step j - 1 runs beside the first phases of step j, which for a job that
    // has just stopped are in vain.  stop[j & 1]: jobs that take no step j.
    const int ph = j & 1;
    auto finish = [&]() {  // the last block's first warp takes the first job, and so on
      __syncthreads();     // sm is free
      if (warp == 0)
        for (int i = nblk - 1 - blk; i < n; i += nblk) {
          DevInst& S = st[i];
          const bool stop = S.stop[ph ^ 1] ? true : step_finish(S, j - 1, sm.finish);
          if (lane == 0) S.stop[ph] = stop;
        }
      __syncthreads();
    };
    auto was_live = [&](const DevInst& S) { return !S.stop[j > 0 ? ph ^ 1 : ph]; };
    auto live = [&](const DevInst& S) { return !S.stop[ph]; };
    const bool traces = border && !own_trace;
    const bool beside = workers < nblk && !traces;  // the last block finishes beside apply and dots
    if (j > 0 && !beside) finish();
    if (j == steps) {
      if (beside) finish();
      return;
    }
    if (traces) {
      for (int i = blk; i < n; i += nblk)
        if (was_live(st[i]) && st[i].border) {
          const double2 a = step_trace<T2>(st[i], j);
          if (threadIdx.x == 0) st[i].alpha = a;
          __syncthreads();
        }
      if (!grid_sync(bar, target)) return;
    }
    if (own_trace && blk < workers) {
      const double2 a = step_trace<T2>(fixed, j);
      if (threadIdx.x == 0) tr = a;
      __syncthreads();
    }
    // items first, first + step, ... of S by this warp
    auto apply = [&](const DevInst& S, int first, int step, int count) {
      const T2* x = (const T2*)S.V + (long long)j * S.ldv;
      const double2* alpha = !S.border ? nullptr : own_trace ? &tr : one ? &st[0].alpha : &S.alpha;
      if constexpr (F32)
        strip_apply32<false>(S, first, step, count, x, (float2*)S.w, alpha);
      else
        for (int k = 0; k < count && first + k * step < S.p64.nitems; ++k)
          strip_apply<false>(S, first + k * step, x, (double2*)S.w, S.scale, alpha);
    };
    if (one) {  // one item per warp, spread over the blocks first
      if (blk < workers) apply(fixed, blk + workers * warp, workers * (kRT / 32), 1 << 30);
    } else {
      for (int t = blk; t < nitem; t += nblk) {
        DevInst& S = st[item_inst[t]];
        if (was_live(S))
          apply(S, item_local[t] * kBlockItems * (F32 ? kRounds32 : 1) + warp, kBlockItems, F32 ? kRounds32 : 1);
      }
    }
    grid_arrive(bar, target);
    if (beside && blk == workers && j > 0) finish();
    if (!grid_wait(bar, target)) return;
    bool any = one;
    for (int i = threadIdx.x; !one && i < n; i += kRT) any = any || live(st[i]);
    if (!__syncthreads_or(any)) return;  // uniform over the grid
    auto dots = [&](bool second) {
      for (int c = blk; c < nchunk; c += nblk) {
        const int inst = one ? 0 : chunk_inst[c];
        if (!one && (!live(st[inst]) || (second && !st[inst].reorth))) continue;
        const DevInst& S = job(inst);
        if constexpr (F32)
          step_dot32<kBatchChunkSmall, 8>(S, j + 1, c, partv, second ? nullptr : part, sm.dot32);
        else
          step_dot64(S, j + 1, c, partv, second ? nullptr : part, sm.dot64);
      }
    };
    auto finals = [&](bool second) {  // one warp per (job, column), spread over the blocks
      for (int t = blk + nblk * warp; t < n * (j + 1); t += nblk * (kRT / 32)) {
        const int i = t / (j + 1), k = t - i * (j + 1);
        if (!one && (!live(st[i]) || (second && !st[i].reorth) || nchunks[i] <= kFewChunks)) continue;
        const DevInst& S = job(i);
        const double2 v = warp_chunk_sum(partv, S.chunk_begin, one ? nc0 : nchunks[i], S.pstride, k);
        if (lane == 0) (second ? S.hB : S.hA)[k] = v;
      }
    };
    // projections of the chunk's job into sm: of a job of few chunks summed here (its first
    // chunk's block keeps them for the finish), otherwise read
    auto projections = [&](const DevInst& S, int inst, int c, bool second, auto* h) {
      double2* keep = second ? S.hB : S.hA;
      auto put = [&](int k, double2 v) {
        if constexpr (F32)
          h[k] = make_float2((float)v.x, (float)v.y);
        else
          h[k] = v;
      };
      const int nc = one ? nc0 : nchunks[inst];
      if (nc <= kFewChunks) {
        for (int k = threadIdx.x; k < 2 * (j + 1); k += kRT) {
          const double v = few_chunk_sum(partv, S.chunk_begin, nc, S.pstride, k);
          if (c == S.chunk_begin) reinterpret_cast<double*>(keep)[k] = v;
          if constexpr (F32)
            reinterpret_cast<float*>(h)[k] = (float)v;
          else
            reinterpret_cast<double*>(h)[k] = v;
        }
      } else {
        for (int k = threadIdx.x; k <= j; k += kRT) put(k, keep[k]);
      }
      __syncthreads();
    };
    auto update = [&](bool second) {
      for (int c = blk; c < nchunk; c += nblk) {
        const int inst = one ? 0 : chunk_inst[c];
        if (!one && (!live(st[inst]) || (second && !st[inst].reorth))) continue;
        const DevInst& S = job(inst);
        if constexpr (F32) {
          projections(S, inst, c, second, sm.axpy32.h);
          step_axpy32(S, j + 1, c, second ? part : part1, sm.axpy32);
        } else {
          projections(S, inst, c, second, sm.axpy64.h);
          step_axpy64(S, j + 1, c, second ? part : part1, sm.axpy64);
        }
      }
    };
    dots(false);
    if (!grid_sync(bar, target)) return;
    if (one && !live(st[0])) return;  // uniform over the grid
    if (many) {
      finals(false);
      if (!grid_sync(bar, target)) return;
    }
    update(false);
    if (!grid_sync(bar, target)) return;
    bool again;
    double rem2 = 0;
    if (one) {
      const StepNorms r = step_norm1(st[0], j + 1, nc0, part, part1, blk == 0);
      again = r.reorth;  // uniform over the grid
      rem2 = r.rem2;
    } else {
      for (int i = blk; i < n; i += nblk)
        if (live(st[i])) step_norm1(st[i], j + 1, nchunks[i], part, part1, true);
      if (!grid_sync(bar, target)) return;
      any = false;
      for (int i = threadIdx.x; i < n; i += kRT) any = any || (live(st[i]) && st[i].reorth);
      again = __syncthreads_or(any);  // uniform over the grid
    }
    if (again) {
      dots(true);
      if (!grid_sync(bar, target)) return;
      if (many) {
        finals(true);
        if (!grid_sync(bar, target)) return;
      }
      update(true);
      if (!grid_sync(bar, target)) return;
      if (one) {
        rem2 = job_norms(fixed, nc0, part, nullptr).x;
        if (blk == 0 && threadIdx.x == 0) st[0].rem2 = rem2;
      } else {
        for (int i = blk; i < n; i += nblk) {
          if (!live(st[i]) || !st[i].reorth) continue;
          const double2 v = job_norms(st[i], nchunks[i], part, nullptr);
          if (threadIdx.x == 0) {
            st[i].rem2 = v.x;
            st[i].inv = inverse_norm(v.x);
          }
        }
        if (!grid_sync(bar, target)) return;
      }
    }
    double f = one ? block_inverse_norm(rem2) : 0.0;
    for (int c = blk; c < nchunk; c += nblk) {
      const int inst = one ? 0 : chunk_inst[c];
      if (!one && !live(st[inst])) continue;
      const DevInst& S = job(inst);
      if (!one) f = st[inst].inv;
      if constexpr (F32)
        step_normalize32(S, j, c, (float)f);
      else
        step_normalize64(S, j, c, f);
    }
    if (!grid_sync(bar, target)) return;
  }
}

// Dense normalized trace vector v = t / (t^H t) in reference coordinates.
__global__ void k_fill_border_vec(const DevSector* __restrict__ sectors, const int* __restrict__ diag_sector,
                                  const long long* __restrict__ diag_index, int ndiag, double2* __restrict__ v) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ndiag; i += gridDim.x * blockDim.x)
    v[diag_index[i]] = make_double2(sectors[diag_sector[i]].border_x, 0.0);
}

template <typename K>
void set_smem(K kernel, size_t bytes, cudaError_t& err) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess && err == cudaSuccess) err = e;
}

}  // namespace

// ---------------------------------------------------------------------------------------
// Job base
// ---------------------------------------------------------------------------------------

Job::~Job() {
  for (void* p : allocs_) cudaFreeAsync(p, s_);
}

void* Job::alloc(size_t b, cudaError_t* err) {
  void* p = nullptr;
  cudaError_t e = cudaMallocAsync(&p, b ? b : 16, s_);
  if (e == cudaErrorMemoryAllocation && reclaim_reserves()) {
    (void)cudaGetLastError();
    e = cudaMallocAsync(&p, b ? b : 16, s_);
  }
  if (e != cudaSuccess) {
    *err = e;
    return nullptr;
  }
  allocs_.push_back(p);
  bytes += b;
  return p;
}

void Job::fail_job(int code, const std::string& m) {
  if (rc == PI_OK) {
    rc = code;
    msg = m;
  }
  finished = true;
}

// ---------------------------------------------------------------------------------------
// Dynamics job
// ---------------------------------------------------------------------------------------

DynamicsJob::DynamicsJob(pi_plan* p, double* state, std::vector<double> times, int nobs, const double* obs,
                         double* values, const pi_expv_opts_t& o, bool single_interval)
    : state_(state), times_(std::move(times)), nobs_(nobs), obs_(obs), values_(values), o_(o), single_(single_interval) {
  plan = p;
  dim = p->host.dim;
}

bool DynamicsJob::setup(cudaStream_t s, int m, bool f32) {
  s_ = s;
  m_engine = m;
  ldh = m + 2;
  mixed_ = f32;
  cudaError_t e = cudaSuccess;
  const size_t es = f32 ? sizeof(float2) : sizeof(double2);
  ldv = basis_stride(dim);
  V = alloc(es * (size_t)ldv * (m + 2), &e);
  w = alloc(es * (size_t)ldv, &e);
  if (e == cudaSuccess) e = cudaMemsetAsync(V, 0, es * (size_t)ldv * (m + 2), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(w, 0, es * (size_t)ldv, s);
  cur_ = (double2*)alloc(sizeof(double2) * dim, &e);
  trial_ = (double2*)alloc(sizeof(double2) * dim, &e);
  if (nobs_ > 0 && mixed_) obsz_ = (double2*)alloc(sizeof(double2) * dim * nobs_, &e);
  if (e != cudaSuccess) return false;
  const DevicePlan& dp = plan->dev;
  if (mixed_) {
    // population coordinates: z = sqrt(f) x; observables dot(O, x) = dot(O / sqrt(f), z)
    e = x_to_z_f64(dp, (const double2*)state_, cur_, 1.0, s);
    for (int o = 0; o < nobs_ && e == cudaSuccess; ++o)
      e = z_to_x_f64(dp, (const double2*)obs_ + (size_t)o * dim, obsz_ + (size_t)o * dim, 1.0, 0, s);
  } else {
    e = cudaMemcpyAsync(cur_, state_, sizeof(double2) * dim, cudaMemcpyDeviceToDevice, s);
  }
  if (e != cudaSuccess) return false;
  obs_pending_ = nobs_ > 0 ? 0 : -1;
  need_norm_ = true;
  return true;
}

unsigned DynamicsJob::stage1(DevInst& d, double2* coef) {
  unsigned f = 0;
  if (obs_pending_ >= 0) {
    d.nob = nobs_;
    d.ob = mixed_ ? obsz_ : (const double2*)obs_;
    d.obx = cur_;
    f |= S1_OBS;
  }
  if (pending_trial_) {
    d.cout = trial_;
    d.ccount = (int)coef_.size();
    d.cacc = 0;
    for (size_t k = 0; k < coef_.size(); ++k) coef[k] = make_double2(coef_[k].real(), coef_[k].imag());
    d.nrm0 = trial_;
    f |= S1_COMBINE | S1_NORM;
  } else if (need_norm_) {
    d.nrm0 = cur_;
    f |= S1_NORM;
  }
  return f;
}

void DynamicsJob::begin_interval() {
  // Zero-length intervals keep the state; their saved values equal the previous ones.
  while (interval_ < (int)times_.size() && times_[interval_] == times_[interval_ - 1]) {
    if (nobs_ > 0) {
      if (obs_pending_ >= 0)
        zero_copies_.push_back(interval_);
      else
        std::memcpy(values_ + (size_t)interval_ * nobs_ * 2, values_ + (size_t)(interval_ - 1) * nobs_ * 2,
                    sizeof(double) * 2 * nobs_);
    }
    ++interval_;
  }
  if (interval_ >= (int)times_.size()) {
    if (obs_pending_ < 0) finished = true;
    return;
  }
  const double dt = times_[interval_] - times_[interval_ - 1];
  total_ = std::abs(dt);
  direction_ = dt < 0 ? -1.0 : 1.0;
  hmax_ = o_.maximum_step > 0 ? o_.maximum_step : total_;
  hmin_ = o_.minimum_step > 0 ? o_.minimum_step : 0.0;
  const double h0 = o_.initial_step > 0 ? o_.initial_step : hmax_;
  hmax_ = std::min(hmax_, total_);
  h_ = std::min(h0, hmax_);
  if (hmin_ > hmax_) return fail_job(PI_ERR_INVALID_ARGUMENT, "minimum_step must not exceed the effective maximum step");
  if (h0 < hmin_) return fail_job(PI_ERR_INVALID_ARGUMENT, "initial_step must not be smaller than minimum_step");
  reached_ = 0.0;
  attempts_ = 0;
  have_ = false;
  attempt();
}

// One trial of krylov_expv!'s loop: factorize if needed, else project again.
void DynamicsJob::attempt() {
  if (attempts_ >= o_.max_steps) {
    char m[200];
    std::snprintf(m, sizeof(m), "adaptive Krylov exponential action reached time %.17g of %.17g after %d attempts",
                  direction_ * reached_, direction_ * total_, attempts_);
    converged_ = false;
    return fail_job(PI_ERR_NOT_CONVERGED, m);
  }
  ++attempts_;
  ++trials_;
  h_ = std::min(h_, total_ - reached_);
  if (!have_)
    want_factor_ = true;
  else
    project();
}

bool DynamicsJob::cycle(DevInst& d) {
  if (!want_factor_ || finished) return false;
  want_factor_ = false;
  ++factorizations_;
  have_ = true;
  beta_ = cur_norm_;
  enlarged_ = false;
  next_rem_ = 0.0;
  if (!std::isfinite(beta_)) {
    fail_job(PI_ERR_INVALID_ARGUMENT, "exponential-action state is not finite");
    return false;
  }
  if (beta_ == 0.0) {
    zero_ = true;
    completed_ = true;
    k_ = q_ = 0;
    project();
    return false;
  }
  zero_ = false;
  d.v0 = cur_;
  d.v0norm = beta_;
  d.m = (int)std::min<long long>(m_engine, dim);
  d.coords = mixed_ ? 1 : 0;
  d.coefb = mixed_ ? (const void*)plan->dev.coef32z : (const void*)plan->dev.coef64;
  d.border = 0;
  d.givens = 0;
  d.scale = 1.0;
  d.tol = 0.0;
  d.j = 0;
  d.done = 0;
  return true;
}

bool DynamicsJob::after_cycle(const DevInst& r, const double2* rec, DevInst& d) {
  const int k = r.kdone;
  const double* image = (const double*)(rec + (size_t)(m_engine + 4) * ldh);
  applications_ += k;
  const double breakfactor = std::sqrt(std::numeric_limits<double>::epsilon());
  const double rem_last = rec[(size_t)(k - 1) * ldh + k].x;
  const bool exact = rem_last == 0.0 || (long long)k == dim;
  bool near = false;
  for (int jj = 0; jj < k; ++jj) {
    const double rem = rec[(size_t)jj * ldh + jj + 1].x;
    if (!std::isfinite(rem)) {
      fail_job(PI_ERR_INVALID_ARGUMENT, "exponential-action Arnoldi remainder is not finite");
      return false;
    }
    if (!std::isfinite(image[jj])) {
      fail_job(PI_ERR_INVALID_ARGUMENT, "exponential-action Arnoldi image is not finite");
      return false;
    }
    if (jj < k - 1 || !exact) near |= rem <= breakfactor * std::max(image[jj], std::numeric_limits<double>::min());
  }
  k_ = k;
  q_ = k + (exact ? 0 : 1);
  S_.assign((size_t)q_ * q_, std::complex<double>(0, 0));
  for (int l = 0; l < k; ++l)
    for (int i = 0; i < k; ++i)
      S_[(size_t)l * q_ + i] = std::complex<double>(rec[(size_t)l * ldh + i].x, rec[(size_t)l * ldh + i].y);
  if (!exact) S_[(size_t)(k - 1) * q_ + k] = std::complex<double>(rem_last, 0.0);
  completed_ = exact;
  if (!exact && near) {
    d.coords = mixed_ ? 1 : 0;
    d.coefb = mixed_ ? (const void*)plan->dev.coef32z : (const void*)plan->dev.coef64;
    d.scale = 1.0;
    d.m = k + 1;
    d.j = k;
    d.done = 0;
    return true;
  }
  project();
  return false;
}

void DynamicsJob::after_enlarge(const DevInst& r, const double2* rec) {
  (void)r;
  const int col = q_ - 1;
  const double* image = (const double*)(rec + (size_t)(m_engine + 4) * ldh);
  for (int i = 0; i < q_; ++i)
    S_[(size_t)col * q_ + i] += std::complex<double>(rec[(size_t)col * ldh + i].x, rec[(size_t)col * ldh + i].y);
  next_rem_ = rec[(size_t)col * ldh + q_].x;
  applications_ += 1;
  if (!std::isfinite(next_rem_))
    return fail_job(PI_ERR_INVALID_ARGUMENT, "exponential-action enlarged Arnoldi remainder is not finite");
  if (!std::isfinite(image[col]))
    return fail_job(PI_ERR_INVALID_ARGUMENT, "exponential-action enlarged Arnoldi image is not finite");
  enlarged_ = true;
  completed_ = ((long long)q_ == dim) || next_rem_ == 0.0;
  project();
}

// _expv_project_factorization! (krylov_extensions.jl:1403-1426).
void DynamicsJob::project() {
  pending_trial_ = true;
  coef_.clear();
  if (zero_) {
    err_ = 0.0;
    return;
  }
  const double h = direction_ * h_;
  CMat A(q_);
  for (int i = 0; i < q_; ++i)
    for (int l = 0; l < q_; ++l) A(i, l) = h * S_[(size_t)l * q_ + i];
  std::vector<std::complex<double>> E;
  try {
    E = expm_column(A);
  } catch (const std::exception& ex) {
    return fail_job(PI_ERR_INVALID_ARGUMENT, std::string("exponential of the projected operator: ") + ex.what());
  }
  const int cc = enlarged_ ? q_ : k_;
  coef_.resize(cc);
  for (int i = 0; i < cc; ++i) coef_[i] = beta_ * E[i];
  if (completed_)
    err_ = 0.0;
  else if (enlarged_)
    err_ = beta_ * std::abs(h) * next_rem_ * std::abs(E[q_ - 1]);
  else
    err_ = beta_ * std::abs(E[k_]);
}

void DynamicsJob::interval_done() {
  if (nobs_ > 0) obs_pending_ = interval_;
  reached_time_ = times_[interval_];
  ++interval_;
  begin_interval();
}

void DynamicsJob::after_stage1(const double* out) {
  if (obs_pending_ >= 0) {
    const int i = obs_pending_;
    for (int o = 0; o < nobs_; ++o) {
      values_[((size_t)i * nobs_ + o) * 2] = out[4 + 2 * o];
      values_[((size_t)i * nobs_ + o) * 2 + 1] = out[5 + 2 * o];
    }
    obs_pending_ = -1;
    // saved times after zero-length intervals repeat these values
    for (int z : zero_copies_)
      std::memcpy(values_ + (size_t)z * nobs_ * 2, values_ + (size_t)i * nobs_ * 2, sizeof(double) * 2 * nobs_);
    zero_copies_.clear();
    if (interval_ >= (int)times_.size() && !pending_trial_ && !want_factor_ && !need_norm_) finished = true;
  }
  if (need_norm_) {
    need_norm_ = false;
    cur_norm_ = std::sqrt(out[0]);
    begin_interval();
    return;
  }
  if (!pending_trial_) return;
  pending_trial_ = false;
  const double error = err_;
  double trial_norm = std::sqrt(out[0]);
  const bool finite = std::isfinite(trial_norm) && std::isfinite(error);
  if (!finite) {
    trial_norm = cur_norm_;
    if (!std::isfinite(trial_norm)) return fail_job(PI_ERR_INVALID_ARGUMENT, "exponential-action state is not finite");
  }
  const double localtol = (h_ / total_) * (o_.atol + o_.rtol * trial_norm);
  if (!std::isfinite(localtol))
    return fail_job(PI_ERR_INVALID_ARGUMENT,
                    "exponential-action local tolerance overflowed; rescale the state or use wider precision");
  const bool accept = finite && (completed_ || error <= localtol);
  if (accept) {
    std::swap(cur_, trial_);
    cur_norm_ = trial_norm;
    const double remaining = total_ - reached_;
    const double next = (h_ == remaining) ? total_ : reached_ + h_;
    if (!(next > reached_))
      return fail_job(PI_ERR_INVALID_ARGUMENT,
                      "exponential-action time step no longer advances; use fewer steps or wider precision");
    reached_ = next;
    ++accepted_;
    error_sum_ += error;
    have_ = false;
  } else {
    ++rejected_;
  }
  double factor;
  if (!finite)
    factor = 0.2;
  else if (completed_)
    factor = 5.0;
  else if (error == 0.0)
    factor = 2.0;
  else {
    factor = o_.safety * std::pow(localtol / error, 1.0 / (double)std::max(k_, 1));
    factor = std::min(std::max(factor, 0.2), 5.0);
  }
  if (!accept) factor = std::min(factor, 0.5);
  const double hnew = std::min(hmax_, h_ * factor);
  if (!accept && (hnew < hmin_ || hnew == 0.0 || (reached_ > 0.0 && reached_ + hnew == reached_))) {
    char m[200];
    std::snprintf(m, sizeof(m), "adaptive Krylov exponential action reached time %.17g of %.17g after %d attempts",
                  direction_ * reached_, direction_ * total_, attempts_);
    converged_ = false;
    return fail_job(PI_ERR_NOT_CONVERGED, m);
  }
  h_ = std::max(hnew, hmin_);
  if (reached_ < total_)
    attempt();
  else
    interval_done();
}

void DynamicsJob::finish(cudaStream_t s) {
  if (mixed_)
    z_to_x_f64(plan->dev, cur_, (double2*)state_, 1.0, 0, s);
  else
    cudaMemcpyAsync(state_, cur_, sizeof(double2) * dim, cudaMemcpyDeviceToDevice, s);
}

pi_expv_info_t DynamicsJob::info() const {
  pi_expv_info_t I;
  std::memset(&I, 0, sizeof(I));
  I.converged = rc == PI_OK && converged_;
  I.reached_time = single_ ? direction_ * reached_ : reached_time_;
  I.accepted_steps = accepted_;
  I.rejected_steps = rejected_;
  I.operator_applications = applications_;
  I.arnoldi_factorizations = factorizations_;
  I.trial_evaluations = trials_;
  I.estimated_error = error_sum_;
  return I;
}

// ---------------------------------------------------------------------------------------
// Steady-state job
// ---------------------------------------------------------------------------------------

SteadyJob::SteadyJob(pi_plan* p, double* x, const pi_gmres_opts_t& o, unsigned long long seed, bool host_probes)
    : x_((double2*)x), o_(o), seed_(seed), host_probes_(host_probes) {
  plan = p;
  dim = p->host.dim;
  bordered = true;
}

bool SteadyJob::setup(cudaStream_t s, int m, bool f32) {
  s_ = s;
  m_engine = m;
  ldh = m + 2;
  mixed_ = f32;
  m_ = (int)std::min<long long>(std::min(o_.krylovdim, m), dim);
  cudaError_t e = cudaSuccess;
  const size_t es = f32 ? sizeof(float2) : sizeof(double2);
  ldv = basis_stride(dim);
  V = alloc(es * (size_t)ldv * (m + 2), &e);
  w = alloc(es * (size_t)ldv, &e);
  if (e == cudaSuccess) e = cudaMemsetAsync(V, 0, es * (size_t)ldv * (m + 2), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(w, 0, es * (size_t)ldv, s);
  b_ = (double2*)alloc(sizeof(double2) * dim, &e);
  r_ = (double2*)alloc(sizeof(double2) * dim, &e);
  ay_ = (double2*)alloc(sizeof(double2) * dim, &e);
  if (e != cudaSuccess) return false;
  const DevicePlan& dp = plan->dev;
  e = cudaMemsetAsync(b_, 0, sizeof(double2) * dim, s);
  if (e == cudaSuccess) {
    const int grid = std::max(1, std::min(608, (dp.ndiag + 255) / 256));
    k_fill_border_vec<<<grid, 256, 0, s>>>(dp.sectors, dp.diag_sector, dp.diag_index, dp.ndiag, b_);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && !o_.use_initial) e = cudaMemcpyAsync(x_, b_, sizeof(double2) * dim, cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) return false;
  if (host_probes_ && o_.operator_scale <= 0) {
    // krylov.jl:156-169 draws three complex normal probes from a seeded generator
    probes_ = (double2*)alloc(sizeof(double2) * dim * 3, &e);
    if (e != cudaSuccess) return false;
    std::vector<double2> h((size_t)dim * 3);
    std::mt19937_64 rng(seed_);
    std::normal_distribution<double> nd(0.0, 1.0);
    // same expression as the host-driven solver (argument evaluation order included)
    for (size_t i = 0; i < h.size(); ++i) h[i] = make_double2(nd(rng) * M_SQRT1_2, nd(rng) * M_SQRT1_2);
    e = cudaMemcpyAsync(probes_, h.data(), sizeof(double2) * h.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // h is released on return
    if (e != cudaSuccess) return false;
  }
  state_ = INIT;
  return true;
}

unsigned SteadyJob::stage1(DevInst& d, double2* coef) {
  switch (state_) {
    case INIT:
      d.nrm0 = b_;
      return S1_NORM;
    case SCALE:
      if (probes_) {
        const double2* pr = probes_ + (size_t)probe_ * dim;
        d.ax = pr;
        d.nrm0 = pr;
      } else {
        d.probe = r_;
        d.seed = seed_ * 4 + (unsigned long long)probe_;
        d.ax = r_;
        d.nrm0 = r_;
      }
      d.ay = ay_;
      d.aux_scale = 1.0;
      d.aux_border = 0;
      d.nrm1 = ay_;
      return (probes_ ? 0u : S1_PROBE) | S1_AUX | S1_NORM;
    case RESID: {
      unsigned f = 0;
      if (pending_update_) {
        d.cout = x_;
        d.ccount = (int)y_.size();
        d.cacc = 1;
        for (size_t k = 0; k < y_.size(); ++k) coef[k] = make_double2(y_[k].real(), y_[k].imag());
        f |= S1_COMBINE;
        pending_update_ = false;
      }
      d.ax = x_;
      d.ay = ay_;
      d.aux_scale = 1.0 / s_op_;
      d.aux_border = 1;
      d.rb = b_;
      d.rout = r_;
      d.nrm0 = r_;
      return f | S1_AUX | S1_RESID | S1_NORM;
    }
    case FINAL:
      d.ax = x_;
      d.ay = ay_;
      d.aux_scale = 1.0;
      d.aux_border = 0;
      d.nrm0 = ay_;
      d.nrm1 = x_;
      d.tr = x_;
      return S1_AUX | S1_NORM | S1_TRACE;
    default:
      return 0;
  }
}

void SteadyJob::after_stage1(const double* out) {
  switch (state_) {
    case INIT:
      tol_ = o_.atol + o_.rtol * std::sqrt(out[0]);
      if (o_.operator_scale > 0) {
        s_op_ = o_.operator_scale;
        state_ = RESID;
      } else {
        state_ = SCALE;
        probe_ = 0;
        scale_ = 0.0;
      }
      break;
    case SCALE:
      // krylov.jl:156-169: max |L r| / |r| over three complex normal probes
      ++applications_;
      scale_ = std::max(scale_, std::sqrt(out[1]) / std::sqrt(out[0]));
      if (++probe_ == 3) {
        s_op_ = scale_;
        if (!(std::isfinite(s_op_) && s_op_ > 0))
          return fail_job(PI_ERR_INVALID_ARGUMENT,
                          "operator_scale must be finite and positive; a numerically zero Liouvillian does not define "
                          "a unique trace-fixed Krylov solve");
        state_ = RESID;
      }
      break;
    case RESID:
      ++applications_;
      beta_ = std::sqrt(out[0]);
      linear_residual_ = beta_;
      if (beta_ <= tol_) {
        gm_converged_ = true;
        state_ = FINAL;
      } else if (iterations_ >= o_.maxiter || (mixed_ && refinements_ >= std::max(1, o_.max_refinements))) {
        state_ = FINAL;
      } else {
        if (mixed_) ++refinements_;
        want_cycle_ = true;
      }
      break;
    case FINAL: {
      ++applications_;
      const double residual = std::sqrt(out[0]);
      const double normalized = residual / s_op_;
      const double xn = std::sqrt(out[1]);
      const double terr = std::abs(std::complex<double>(out[2], out[3]) - std::complex<double>(1, 0));
      const double tol = o_.atol + o_.rtol * std::max(xn, 1.0);
      std::memset(&info_, 0, sizeof(info_));
      info_.converged = gm_converged_ && normalized <= tol && terr <= o_.atol + o_.rtol;
      info_.iterations = iterations_;
      info_.restarts = restarts_;
      info_.refinements = refinements_;
      info_.operator_applications = applications_;
      info_.residual = residual;
      info_.normalized_residual = normalized;
      info_.trace_error = terr;
      info_.operator_scale = s_op_;
      info_.linear_residual = linear_residual_;
      state_ = DONE;
      finished = true;
      if (!info_.converged) {
        char m[256];
        std::snprintf(m, sizeof(m),
                      "matrix-free Krylov steady-state solve did not converge in %d iterations; "
                      "normalized_residual=%.3e, trace_error=%.3e",
                      iterations_, normalized, terr);
        rc = PI_ERR_NOT_CONVERGED;
        msg = m;
      }
      break;
    }
    default:
      break;
  }
}

bool SteadyJob::cycle(DevInst& d) {
  if (!want_cycle_ || finished) return false;
  want_cycle_ = false;
  d.v0 = r_;
  d.v0norm = beta_;
  d.m = std::min(m_, o_.maxiter - iterations_);
  d.border = 1;
  d.givens = 1;
  d.scale = 1.0 / s_op_;
  d.coords = 0;
  d.coefb = mixed_ ? (const void*)plan->dev.coef32x : (const void*)plan->dev.coef64;
  // FP32 inner solves stop at a relative reduction they can resolve; the FP64 outer
  // residual restores the rest.
  d.tol = mixed_ ? std::max(tol_ * 0.5, 1e-5 * beta_) : tol_;
  d.j = 0;
  d.done = 0;
  return true;
}

bool SteadyJob::after_cycle(const DevInst& r, const double2* rec, DevInst&) {
  const int k = r.kdone;
  iterations_ += k;
  applications_ += k;
  if (k == 0) {
    state_ = FINAL;
    return false;
  }
  const double2* g = rec + (size_t)(m_engine + 1) * ldh;
  y_.assign(k, std::complex<double>(0, 0));
  for (int i = k - 1; i >= 0; --i) {
    std::complex<double> s(g[i].x, g[i].y);
    for (int jj = i + 1; jj < k; ++jj) {
      const double2 h = rec[(size_t)jj * ldh + i];
      s -= std::complex<double>(h.x, h.y) * y_[jj];
    }
    const double2 hd = rec[(size_t)i * ldh + i];
    if (hd.x == 0.0 && hd.y == 0.0) {
      fail_job(PI_ERR_NOT_CONVERGED, "singular GMRES triangular factor");
      return false;
    }
    y_[i] = s / std::complex<double>(hd.x, hd.y);
  }
  ++restarts_;
  pending_update_ = true;
  state_ = RESID;
  return false;
}

// ---------------------------------------------------------------------------------------
// Engine
// ---------------------------------------------------------------------------------------

Engine::Engine(int device, int krylovdim, bool f32, bool use_graphs)
    : device_(device), m_(krylovdim), f32_(f32), graphs_(use_graphs) {
  chk(cudaSetDevice(device));
  chk(cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking));
  // Job workspaces come from the device's default memory pool; keep freed memory in the
  // pool so that admitting the next requests does not go back to the driver.
  cudaMemPool_t pool = nullptr;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess && pool) {
    unsigned long long keep = ~0ULL;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  const size_t smem64 = 3 * kWinElems * sizeof(double2);
  const size_t smem32 = 3 * kWinElems * sizeof(float2);
  set_smem(k_bapply<double, true>, smem64, err);
  set_smem(k_bapply<double, false>, smem64, err);
  set_smem(k_bapply<float, false>, smem32, err);
  set_smem(k_bapply_persist, kSepSmemBytes, err);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cycle_max_, f32 ? k_cycle<true> : k_cycle<false>, kRT, 0) !=
      cudaSuccess) {
    cycle_max_ = 0;
    (void)cudaGetLastError();  // no one-launch cycles; the error is not the engine's
  }
  chk(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device));
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&persist_max_, k_bapply_persist, kApplyThreads,
                                                    kSepSmemBytes) != cudaSuccess) {
    persist_max_ = 0;
    (void)cudaGetLastError();  // no persistent schedule; the error is not the engine's
  }
  rec_stride_ = (size_t)(m_ + 5) * (m_ + 2);
}

Engine::~Engine() {
  if (graph_) cudaGraphExecDestroy(graph_);
  if (s_) cudaStreamSynchronize(s_);
  for (void* p : {st_, tile_inst_, tile_local_, strip_inst_, strip_local_, bar_, again_, chunk_inst_, nchunks_, part1_, partv_, hab_, rec_, out_, coefs_})
    if (p) cudaFree(p);
  for (void* p : {st_h_, st_dl_, rec_h_, out_h_, coefs_h_})
    if (p) cudaFreeHost(p);
  if (s_) cudaStreamDestroy(s_);
}

void Engine::reserve(void** p, size_t* cap, size_t bytes, bool pinned) {
  if (bytes <= *cap && *p) return;
  chk(cudaStreamSynchronize(s_));
  if (*p) {
    if (pinned)
      cudaFreeHost(*p);
    else
      cudaFree(*p);
    *p = nullptr;
  }
  const size_t nb = std::max(bytes + bytes / 2, (size_t)256);
  chk(pinned ? cudaMallocHost(p, nb) : cudaMalloc(p, nb));
  *cap = *p ? nb : 0;
}

void Engine::add(Job* j) {
  jobs_.push_back(j);
  dirty_ = true;
}

std::vector<Job*> Engine::retire() {
  std::vector<Job*> done, keep;
  for (Job* j : jobs_) (j->finished ? done : keep).push_back(j);
  if (!done.empty()) {
    jobs_.swap(keep);
    dirty_ = true;
  }
  return done;
}

void Engine::rebuild() {
  const int n = (int)jobs_.size();
  const size_t nn = std::max(n, 1);
  const int pstride = std::max(m_ + 2, kBatchMaxObs);  // chunk partials: basis columns or observables
  // Chunk size: large chunks amortise the per-block reductions; when the active jobs hold
  // fewer elements than about eight large chunks per SM, small chunks keep the GPU full.
  long long total_elems = 0;
  for (int i = 0; i < n; ++i) total_elems += jobs_[i]->dim;
  chunk_ = total_elems >= 8LL * 152 * kBatchChunk ? kBatchChunk : kBatchChunkSmall;
  // the trace of each step's input column is only needed by bordered (steady-state) cycles
  any_border_ = false;
  for (int i = 0; i < n; ++i) any_border_ = any_border_ || jobs_[i]->bordered;
  std::vector<int> ti, tl, si, sl, ci, nc(n);
  std::vector<Planes64> p64(n);
  std::vector<SplitPlanes> p32(n, SplitPlanes{nullptr, nullptr, nullptr, nullptr, 0});
  std::vector<StripItems> it32(n);
  bool canonical = true;  // every job steps by strips
  for (int i = 0; i < n; ++i) {
    pi_plan* plan = jobs_[i]->plan;
    // Step applies of canonical plans run over strip blocks, of other plans over tiles.  FP32
    // dynamics cycles run in population coordinates, steady-state cycles in reference ones.
    int strips = 0;
    if (f32_) {
      if (plan->dev.canon && em_split_planes(plan, jobs_[i]->bordered ? 0 : 1, &p32[i]) == PI_OK)
        it32[i] = strip_items(plan, s_);
      else
        p32[i] = SplitPlanes{nullptr, nullptr, nullptr, nullptr, 0};
      strips = it32[i].n;
    } else {
      p64[i] = planes64(plan, PI_COORDS_REFERENCE, s_);
      strips = p64[i].nitems;
    }
    const int ntiles = plan->dev.ntiles;
    const int per = f32_ ? kBlockItems * kRounds32 : kBlockItems;
    const int nstrip = strips ? (strips + per - 1) / per : ntiles;
    canonical = canonical && strips > 0;
    for (int t = 0; t < ntiles; ++t) {
      ti.push_back(i);
      tl.push_back(t);
    }
    for (int t = 0; t < nstrip; ++t) {
      si.push_back(i);
      sl.push_back(t);
    }
    const int chunk = f32_ ? chunk_ : chunk64(jobs_[i]->dim);
    nc[i] = (int)((jobs_[i]->dim + chunk - 1) / chunk);
  }
  reserve(&hab_, &hab_cap_, sizeof(double2) * 2 * kMaxDots * nn, false);
  reserve(&rec_, &rec_cap_, sizeof(double2) * rec_stride_ * nn, false);
  reserve(&out_, &out_cap_, sizeof(double) * kOutSlots * nn, false);
  reserve(&coefs_, &coefs_cap_, sizeof(double2) * (m_ + 2) * nn, false);
  base_.assign(n, DevInst());
  for (int i = 0; i < n; ++i) {
    Job* J = jobs_[i];
    const DevicePlan& dp = J->plan->dev;
    DevInst& d = base_[i];
    std::memset(&d, 0, sizeof(d));
    d.sectors = dp.sectors;
    d.terms = dp.terms;
    d.tiles = dp.tiles;
    d.coef64 = dp.coef64;
    d.coefb = f32_ ? (const void*)dp.coef32x : (const void*)dp.coef64;
    d.diag_sector = dp.diag_sector;
    d.diag_index = dp.diag_index;
    d.dim = J->dim;
    d.ldv = J->ldv;
    d.ndiag = dp.ndiag;
    d.chunk_begin = (int)ci.size();
    d.chunk = f32_ ? chunk_ : chunk64(J->dim);
    d.pstride = pstride;
    d.planes = p32[i];
    d.pwhich = J->bordered ? 0 : 1;
    d.items32 = it32[i].items;
    d.nitems32 = it32[i].n;
    d.p64 = p64[i];
    for (int c = 0; c < nc[i]; ++c) ci.push_back(i);
    d.V = J->V;
    d.w = J->w;
    d.hA = (double2*)hab_ + (size_t)i * 2 * kMaxDots;
    d.hB = d.hA + kMaxDots;
    double2* rec = (double2*)rec_ + (size_t)i * rec_stride_;
    d.H = rec;
    d.g = rec + (size_t)(m_ + 1) * (m_ + 2);
    d.csn = rec + (size_t)(m_ + 2) * (m_ + 2);
    d.image = (double*)(rec + (size_t)(m_ + 4) * (m_ + 2));
    d.ldh = m_ + 2;
    d.ccoef = (const double2*)coefs_ + (size_t)i * (m_ + 2);
    d.out = (double*)out_ + (size_t)i * kOutSlots;
    d.scale = 1.0;
    d.aux_scale = 1.0;
    d.done = 1;
  }
  total_tiles_ = (int)ti.size();
  total_strips_ = (int)si.size();
  cycle_kernel_ = canonical && n > 0 && total_elems <= kCycleElems && cycle_max_ > 0 && sm_count_ > 0;
  total_chunks_ = (int)ci.size();
  plan_cycle();
  reserve(&st_, &st_cap_, sizeof(DevInst) * nn, false);
  reserve(&tile_inst_, &tile_inst_cap_, sizeof(int) * std::max<size_t>(ti.size(), 1), false);
  reserve(&tile_local_, &tile_local_cap_, sizeof(int) * std::max<size_t>(tl.size(), 1), false);
  reserve(&strip_inst_, &strip_inst_cap_, sizeof(int) * std::max<size_t>(si.size(), 1), false);
  reserve(&strip_local_, &strip_local_cap_, sizeof(int) * std::max<size_t>(sl.size(), 1), false);
  reserve(&bar_, &bar_cap_, sizeof(GridBar), false);
  reserve(&again_, &again_cap_, sizeof(int), false);
  chk(cudaMemsetAsync(again_, 0, sizeof(int), s_));
  reserve(&chunk_inst_, &chunk_inst_cap_, sizeof(int) * std::max<size_t>(ci.size(), 1), false);
  reserve(&nchunks_, &nchunks_cap_, sizeof(int) * nn, false);
  reserve(&part1_, &part1_cap_, sizeof(double) * 2 * std::max(total_chunks_, 1), false);
  reserve(&partv_, &partv_cap_, sizeof(double2) * (size_t)pstride * std::max(total_chunks_, 1), false);
  reserve(&st_h_, &st_h_cap_, sizeof(DevInst) * nn, true);
  reserve(&st_dl_, &st_dl_cap_, sizeof(DevInst) * nn, true);
  reserve(&rec_h_, &rec_h_cap_, sizeof(double2) * rec_stride_ * nn, true);
  reserve(&out_h_, &out_h_cap_, sizeof(double) * kOutSlots * nn, true);
  reserve(&coefs_h_, &coefs_h_cap_, sizeof(double2) * (m_ + 2) * nn, true);
  if (!ti.empty()) chk(cudaMemcpyAsync(tile_inst_, ti.data(), sizeof(int) * ti.size(), cudaMemcpyHostToDevice, s_));
  if (!tl.empty()) chk(cudaMemcpyAsync(tile_local_, tl.data(), sizeof(int) * tl.size(), cudaMemcpyHostToDevice, s_));
  if (!si.empty()) chk(cudaMemcpyAsync(strip_inst_, si.data(), sizeof(int) * si.size(), cudaMemcpyHostToDevice, s_));
  if (!sl.empty()) chk(cudaMemcpyAsync(strip_local_, sl.data(), sizeof(int) * sl.size(), cudaMemcpyHostToDevice, s_));
  if (!ci.empty()) chk(cudaMemcpyAsync(chunk_inst_, ci.data(), sizeof(int) * ci.size(), cudaMemcpyHostToDevice, s_));
  if (n) chk(cudaMemcpyAsync(nchunks_, nc.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s_));
  chk(cudaStreamSynchronize(s_));  // the host vectors above go out of scope
  if (graph_) {
    cudaGraphExecDestroy(graph_);
    graph_ = nullptr;
  }
  schedule_chosen_ = cycle_recorded_ = false;
  dirty_ = false;
}

namespace {

// Process-wide schedule setting, choice cache and the record of the last choice.
std::atomic<int> g_apply_schedule{PI_SCHEDULE_AUTO};
std::mutex g_schedule_mu;
std::map<long long, int> g_schedule_cache;  // (device, job-set shape) -> schedule
pi_schedule_info_t g_schedule_info{};

// `rec` (work list, resident limit, candidates) becomes the record of the last choice.
void record_schedule(pi_schedule_info_t rec, int schedule) {
  std::lock_guard<std::mutex> lk(g_schedule_mu);
  rec.choices = g_schedule_info.choices + 1;
  rec.tunings = g_schedule_info.tunings;
  rec.schedule = schedule;
  g_schedule_info = rec;
}

}  // namespace

void Engine::launch_step_apply(int schedule) {
  DevInst* st = (DevInst*)st_;
  const int* ti = (const int*)tile_inst_;
  const int* tl = (const int*)tile_local_;
  if (schedule > 0) {
    const int grid = std::max(1, std::min(total_tiles_, schedule * sm_count_));
    launch(k_bapply_persist, grid, kApplyThreads, kSepSmemBytes, (const DevInst*)st, ti, tl, total_tiles_);
  } else {
    launch(k_bapply<float, false>, total_strips_, kApplyThreads, 3 * kWinElems * sizeof(float2), (const DevInst*)st,
           (const int*)strip_inst_, (const int*)strip_local_);
  }
}

// Picks the FP32 step-apply schedule of the current job set.  Runs on the engine stream
// after the cycle's control blocks and first basis columns are on the device and before the
// cycle's steps are launched or captured: the timed applies write only each running job's
// step column w, which the first step overwrites.
void Engine::choose_apply_schedule() {
  schedule_chosen_ = true;
  apply_schedule_ = PI_SCHEDULE_PER_TILE;
  if (!f32_ || total_tiles_ == 0 || persist_max_ < 1 || sm_count_ < 1) return;
  const int setting = g_apply_schedule.load();
  bool general = false;
  for (const DevInst& d : base_) general = general || d.planes.srow == nullptr;
  int size_class = 0;
  while ((2LL << size_class) <= total_tiles_) ++size_class;
  const long long key = ((long long)device_ << 16) | (size_class << 1) | (general ? 1 : 0);
  pi_schedule_info_t rec{};
  rec.items = total_tiles_;
  rec.resident_max = persist_max_;
  if (setting != PI_SCHEDULE_AUTO) {
    apply_schedule_ = setting > 0 ? std::min(setting, persist_max_) : PI_SCHEDULE_PER_TILE;
  } else {
    bool cached = false;
    {
      std::lock_guard<std::mutex> lk(g_schedule_mu);
      auto it = g_schedule_cache.find(key);
      if (it != g_schedule_cache.end()) {
        apply_schedule_ = std::min(it->second, persist_max_);
        cached = true;
      }
    }
    if (!cached) {
      std::vector<int> cand{PI_SCHEDULE_PER_TILE};
      for (int b = 1; b <= std::min(persist_max_, 7); ++b) cand.push_back(b);
      cudaEvent_t e0 = nullptr, e1 = nullptr;
      chk(cudaEventCreate(&e0));
      chk(cudaEventCreate(&e1));
      constexpr int kReps = 3;
      double best = 0;
      for (size_t c = 0; c < cand.size() && err == cudaSuccess; ++c) {
        launch_step_apply(cand[c]);  // warm-up
        float t[kReps];
        for (int r = 0; r < kReps; ++r) {
          chk(cudaEventRecord(e0, s_));
          launch_step_apply(cand[c]);
          chk(cudaEventRecord(e1, s_));
          chk(cudaEventSynchronize(e1));
          t[r] = 0.f;
          chk(cudaEventElapsedTime(&t[r], e0, e1));
        }
        std::sort(t, t + kReps);
        const double us = 1e3 * t[kReps / 2];
        rec.cand[rec.ncand] = cand[c];
        rec.cand_us[rec.ncand] = us;
        ++rec.ncand;
        if (c == 0 || us < best) {
          best = us;
          apply_schedule_ = cand[c];
        }
      }
      chk(cudaGetLastError());
      if (e0) cudaEventDestroy(e0);
      if (e1) cudaEventDestroy(e1);
      if (err == cudaSuccess) {
        std::lock_guard<std::mutex> lk(g_schedule_mu);
        g_schedule_cache[key] = apply_schedule_;
        ++g_schedule_info.tunings;
      }
    }
  }
  record_schedule(rec, apply_schedule_);
}

// Launches a kernel on the engine stream, or appends it as the next node of the graph under
// construction (explicit kernel nodes, no stream capture: a capture would forbid
// device-wide synchronisation by other host threads, e.g. a serving client).
template <typename... KArgs, typename... Args>
void Engine::launch(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, Args... args) {
  if (!build_) {
    k<<<grid, block, smem, s_>>>(args...);
    return;
  }
  std::tuple<KArgs...> vals(args...);
  void* ptrs[sizeof...(KArgs)];
  fill_ptrs(vals, ptrs, std::index_sequence_for<KArgs...>{});
  cudaKernelNodeParams p{};
  p.func = reinterpret_cast<void*>(k);
  p.gridDim = grid;
  p.blockDim = block;
  p.sharedMemBytes = (unsigned)smem;
  p.kernelParams = ptrs;
  p.extra = nullptr;
  cudaGraphNode_t node = nullptr;
  chk(cudaGraphAddKernelNode(&node, build_, last_ ? &last_ : nullptr, last_ ? 1 : 0, &p));
  if (node) last_ = node;
}

void Engine::arnoldi_step() {
  DevInst* st = (DevInst*)st_;
  const DevInst* cst = st;
  const int* ci = (const int*)chunk_inst_;
  const int* nc = (const int*)nchunks_;
  double* part = (double*)part1_;
  double2* partv = (double2*)partv_;
  const double2* cpartv = partv;
  const int n = (int)jobs_.size();
  const dim3 gfin(n, (m_ + 1 + kRT / 32 - 1) / (kRT / 32));
  const int C = total_chunks_;
  double* npart1 = part + C;  // |w1|^2 partials of the first update (second half of part)
  // Classical Gram-Schmidt with selective reorthogonalisation: the first pass also takes the
  // image norm |w0|^2 and the first update the |w1|^2 partials; the blocks of the second pass
  // return at once for jobs that need none (step_norm1).
  const int* again = (const int*)again_;
  auto grid = [&](int second) { return second ? std::min(C, kSecondPassBlocks) : C; };
  auto dots = [&](int second) {
    double* ipart = second ? nullptr : part;
    if (!f32_)
      launch(k_step_dot64, grid(second), kRT, 0, cst, ci, C, partv, ipart, second ? again : nullptr);
    else if (chunk_ == kBatchChunk)
      launch(k_step_mdot_f32<kBatchChunk>, grid(second), kRT, 0, cst, ci, C, partv, ipart, second ? again : nullptr);
    else
      launch(k_step_mdot_f32<kBatchChunkSmall>, grid(second), kRT, 0, cst, ci, C, partv, ipart,
             second ? again : nullptr);
  };
  auto update = [&](int second) {
    double* out = second ? part : npart1;
    if (f32_)
      launch(k_step_maxpy_f32, grid(second), kRT, 0, cst, ci, C, out, second ? again : nullptr);
    else
      launch(k_step_axpy64, grid(second), kRT, 0, cst, ci, C, out, second ? again : nullptr);
  };
  if (f32_) {
    if (any_border_) launch(k_step_trace<float2>, n, kRT, 0, st);
    launch_step_apply(apply_schedule_);
  } else {
    if (any_border_) launch(k_step_trace<double2>, n, kRT, 0, st);
    launch(k_bapply<double, false>, total_strips_, kApplyThreads, 3 * kWinElems * sizeof(double2), cst,
           (const int*)strip_inst_, (const int*)strip_local_);
  }
  dots(0);
  launch(k_step_first_final, gfin, kRT, 0, st, nc, cpartv);
  update(0);
  launch(k_step_norm, n, kRT, 0, st, nc, (const double*)part, (const double*)npart1, 0, (int*)again_);
  dots(1);
  launch(k_step_mdot_final, gfin, kRT, 0, cst, nc, cpartv);
  update(1);
  launch(k_step_norm, n, kRT, 0, st, nc, (const double*)part, (const double*)npart1, 1, (int*)again_);
  if (f32_)
    launch(k_step_normalize_f32, C, kRT, 0, cst, ci);
  else
    launch(k_step_normalize64, C, kRT, 0, cst, ci);
  launch(k_step_finish, n, 32, 0, st, (int*)again_);
  if (!build_) chk(cudaGetLastError());
}

// The cycle of a small job set in one launch: a block more than its longest work list has entries
// (the finish of a single job), at most what is resident at once.  Up to kMaxCluster blocks are a
// cluster, whose barrier costs less than the grid barrier; larger sets are cooperative launches.
// Sets that would have to fold onto a cluster lose more than that: N = 14 (22 chunks) takes 6.1 ms
// as 23 cooperative blocks and 7.1 as a cluster of 16, N = 16 GMRES 15.7 and 19.6.
static const void* cycle_fn(bool f32) {
  return f32 ? (const void*)k_cycle<true> : (const void*)k_cycle<false>;
}
static cudaLaunchConfig_t cluster_config(int blocks, cudaLaunchAttribute* at) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = blocks;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kRT);
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}
constexpr int kMaxCluster = 16;

void Engine::plan_cycle() {
  cycle_grid_ = std::max(1, std::min(std::max(total_chunks_, total_strips_) + 1, cycle_max_ * sm_count_));
  cycle_cluster_ = cycle_kernel_ && cycle_grid_ > 1 && cycle_grid_ <= kMaxCluster;
  if (!cycle_cluster_) return;
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = cluster_config(cycle_grid_, &at);
  int fit = 0;
  if (cudaFuncSetAttribute(cycle_fn(f32_), cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&fit, cycle_fn(f32_), &cfg) != cudaSuccess) {
    fit = 0;
    (void)cudaGetLastError();  // the cooperative launch serves
  }
  cycle_cluster_ = fit > 0;
}

void Engine::launch_cycle() {
  const int n = (int)jobs_.size();
  const int grid = cycle_grid_;
  DevInst* st = (DevInst*)st_;
  const int *ci = (const int*)chunk_inst_, *si = (const int*)strip_inst_, *sl = (const int*)strip_local_;
  const int* nc = (const int*)nchunks_;
  double2* partv = (double2*)partv_;
  double* part = (double*)part1_;
  GridBar* bar = cycle_cluster_ ? nullptr : (GridBar*)bar_;
  int nn = n, C = total_chunks_, T = total_strips_, steps = m_, border = any_border_ ? 1 : 0;
  chk(cudaMemsetAsync(bar_, 0, sizeof(GridBar), s_));
  void* args[] = {&st, &nn, &ci, &C, &si, &sl, &T, &nc, &partv, &part, &steps, &border, &bar};
  if (cycle_cluster_) {
    cudaLaunchAttribute at{};
    cudaLaunchConfig_t cfg = cluster_config(grid, &at);
    cfg.stream = s_;
    chk(cudaLaunchKernelExC(&cfg, cycle_fn(f32_), args));
    return;
  }
  chk(cudaLaunchCooperativeKernel(cycle_fn(f32_), dim3(grid), dim3(kRT), args, 0, s_));
}

// Steps per graph.  Building and instantiating a graph takes about 1.7 us per node, once per job
// set, and each step has about ten.
constexpr int kGraphSteps = 5;

void Engine::run_cycle_steps() {
  // an explicit step-apply schedule asks for the step kernels
  ran_cycle_ = cycle_kernel_ && (!f32_ || g_apply_schedule.load() == PI_SCHEDULE_AUTO);
  if (ran_cycle_) {
    if (f32_ && !cycle_recorded_) {  // once per job set, like a choice among the step schedules
      pi_schedule_info_t rec{};
      rec.items = total_strips_;
      rec.resident_max = persist_max_;
      record_schedule(rec, PI_SCHEDULE_ONE_LAUNCH);
      cycle_recorded_ = true;
    }
    launch_cycle();
    return;
  }
  if (!schedule_chosen_) choose_apply_schedule();
  if (err != cudaSuccess) return;
  if (!graphs_) {
    for (int j = 0; j < m_; ++j) arnoldi_step();
    return;
  }
  if (!graph_) {
    chk(cudaGraphCreate(&build_, 0));
    last_ = nullptr;
    if (build_) {
      for (int j = 0; j < std::min(m_, kGraphSteps); ++j) arnoldi_step();
      if (err == cudaSuccess) chk(cudaGraphInstantiate(&graph_, build_, 0));
      cudaGraphDestroy(build_);
    }
    build_ = nullptr;
    last_ = nullptr;
    if (err != cudaSuccess) return;
  }
  for (int j = kGraphSteps; j <= std::max(m_, kGraphSteps); j += kGraphSteps) chk(cudaGraphLaunch(graph_, s_));
  for (int j = m_ < kGraphSteps ? 0 : m_ % kGraphSteps; j > 0; --j) arnoldi_step();
}

// f(i) for every job, those in `busy` spread over a few host threads: a cycle's end costs each of
// its jobs about 0.1 ms on the host while the GPU waits.  24 jobs: 2.0 -> 0.5 ms per tick.
template <typename F>
static void for_jobs(const std::vector<char>& busy, const F& f) {
  const int n = (int)busy.size();
  const long count = std::count(busy.begin(), busy.end(), 1);
  const int threads = (int)std::min<long>({count / 2, 8, (long)std::thread::hardware_concurrency()});
  std::atomic<int> next{0};
  std::exception_ptr thrown;
  std::mutex thrown_mu;
  auto work = [&] {
    try {
      for (int i = next++; i < n; i = next++) f(i);
    } catch (...) {  // goes on in the calling thread, as without helpers
      std::lock_guard<std::mutex> lk(thrown_mu);
      if (!thrown) thrown = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  try {
    for (int t = 1; t < threads; ++t) pool.emplace_back(work);
  } catch (const std::system_error&) {  // no further thread to be had: this one does the rest
  }
  work();
  for (std::thread& t : pool) t.join();
  if (thrown) std::rethrow_exception(thrown);
}

bool Engine::tick() {
  if (err != cudaSuccess) return false;
  if (dirty_) rebuild();
  if (err != cudaSuccess) return false;
  const int n = (int)jobs_.size();
  if (n == 0) return true;
  ++ticks;
  DevInst* sth = (DevInst*)st_h_;
  double2* coefh = (double2*)coefs_h_;
  const double* outh = (const double*)out_h_;
  DevInst* st = (DevInst*)st_;
  const int* ci = (const int*)chunk_inst_;
  const int* ti = (const int*)tile_inst_;
  const int* tl = (const int*)tile_local_;
  const int C = total_chunks_;
  // ---- stage 1: vector work and one read
  unsigned flags = 0;
  for (int i = 0; i < n; ++i) {
    sth[i] = base_[i];
    if (!jobs_[i]->finished) flags |= jobs_[i]->stage1(sth[i], coefh + (size_t)i * (m_ + 2));
  }
  if (flags) {
    chk(cudaMemcpyAsync(st_, st_h_, sizeof(DevInst) * n, cudaMemcpyHostToDevice, s_));
    if (flags & S1_COMBINE) {
      chk(cudaMemcpyAsync(coefs_, coefs_h_, sizeof(double2) * (m_ + 2) * n, cudaMemcpyHostToDevice, s_));
      if (f32_)
        k_s1_combine_f32<<<C, kRT, 0, s_>>>(st, ci, (double*)part1_);
      else
        k_s1_combine<<<C, kRT, 0, s_>>>(st, ci, (double*)part1_);
    }
    if (flags & S1_PROBE) k_s1_probe<<<C, kRT, 0, s_>>>(st, ci);
    if (flags & (S1_AUX | S1_TRACE)) k_s1_trace<<<n, kRT, 0, s_>>>(st);
    if (flags & S1_AUX)
      // an FP64 engine's canonical plans by strips, an FP32 engine's by tiles
      k_bapply<double, true><<<f32_ ? total_tiles_ : total_strips_, kApplyThreads, 3 * kWinElems * sizeof(double2),
                               s_>>>(st, f32_ ? ti : (const int*)strip_inst_, f32_ ? tl : (const int*)strip_local_);
    if (flags & S1_RESID) k_s1_resid<<<C, kRT, 0, s_>>>(st, ci);
    bool norms = false;  // beyond those of combinations
    for (int i = 0; i < n; ++i) norms = norms || (sth[i].nrm0 && sth[i].nrm0 != sth[i].cout) || sth[i].nrm1;
    if (norms) k_s1_norm_partial<<<C, kRT, 0, s_>>>(st, ci, (double*)part1_);
    if (flags & S1_OBS) k_s1_obs_partial<<<C, kRT, 0, s_>>>(st, ci, (double2*)partv_);
    if (flags & (S1_NORM | S1_OBS))
      k_s1_final<<<n, kRT, 0, s_>>>(st, (const int*)nchunks_, (const double*)part1_, (const double2*)partv_);
    chk(cudaGetLastError());
    chk(cudaMemcpyAsync(out_h_, out_, sizeof(double) * kOutSlots * n, cudaMemcpyDeviceToHost, s_));
    chk(cudaStreamSynchronize(s_));
    if (err != cudaSuccess) return false;
    for (int i = 0; i < n; ++i)
      if (!jobs_[i]->finished) jobs_[i]->after_stage1(outh + (size_t)i * kOutSlots);
  }
  // ---- stage 3: one Arnoldi cycle for the jobs that need a factorization
  std::vector<char> in_cycle(n, 0);
  bool any = false;
  for (int i = 0; i < n; ++i) {
    sth[i] = base_[i];
    if (!jobs_[i]->finished && jobs_[i]->cycle(sth[i])) {
      in_cycle[i] = 1;
      any = true;
    }
    sth[i].stop[0] = sth[i].stop[1] = sth[i].done;
  }
  if (!any) return err == cudaSuccess;
  ++cycles;
  chk(cudaMemcpyAsync(st_, st_h_, sizeof(DevInst) * n, cudaMemcpyHostToDevice, s_));
  if (f32_)
    k_load_v0<float2><<<C, kRT, 0, s_>>>(st, ci);
  else
    k_load_v0<double2><<<C, kRT, 0, s_>>>(st, ci);
  chk(cudaGetLastError());
  run_cycle_steps();
  steps += m_;
  const DevInst* dl = (const DevInst*)st_dl_;
  const double2* rech = (const double2*)rec_h_;
  chk(cudaMemcpyAsync(st_dl_, st_, sizeof(DevInst) * n, cudaMemcpyDeviceToHost, s_));
  chk(cudaMemcpyAsync(rec_h_, rec_, sizeof(double2) * rec_stride_ * n, cudaMemcpyDeviceToHost, s_));
  GridBar bar{0, 0};
  if (ran_cycle_) chk(cudaMemcpyAsync(out_h_, bar_, sizeof(GridBar), cudaMemcpyDeviceToHost, s_));
  chk(cudaStreamSynchronize(s_));
  if (ran_cycle_) std::memcpy(&bar, out_h_, sizeof(bar));
  if (bar.err) chk(cudaErrorLaunchTimeout);  // a grid barrier gave up waiting
  if (err != cudaSuccess) return false;
  bool enl = false;
  std::vector<char> in_enl(n, 0);
  // the jobs' small dense problems (a matrix exponential each), several jobs at a time
  for_jobs(in_cycle, [&](int i) {
    sth[i] = base_[i];
    in_enl[i] = in_cycle[i] && jobs_[i]->after_cycle(dl[i], rech + (size_t)i * rec_stride_, sth[i]);
  });
  for (int i = 0; i < n; ++i) enl = enl || in_enl[i];
  if (!enl) return err == cudaSuccess;
  // near-breakdown enlargement: one more step for the jobs that asked
  chk(cudaMemcpyAsync(st_, st_h_, sizeof(DevInst) * n, cudaMemcpyHostToDevice, s_));
  arnoldi_step();
  ++steps;
  chk(cudaMemcpyAsync(st_dl_, st_, sizeof(DevInst) * n, cudaMemcpyDeviceToHost, s_));
  chk(cudaMemcpyAsync(rec_h_, rec_, sizeof(double2) * rec_stride_ * n, cudaMemcpyDeviceToHost, s_));
  chk(cudaStreamSynchronize(s_));
  if (err != cudaSuccess) return false;
  for (int i = 0; i < n; ++i)
    if (in_enl[i]) jobs_[i]->after_enlarge(dl[i], rech + (size_t)i * rec_stride_);
  return err == cudaSuccess;
}

int run_single_job(pi_plan* plan, Job* job, int m, bool f32, const char* what) {
  if (plan->engine && (plan->engine_m != m || plan->engine_f32 != f32 || plan->engine->err != cudaSuccess)) {
    delete plan->engine;
    plan->engine = nullptr;
  }
  if (!plan->engine) {
    plan->engine = new Engine(plan->device, m, f32, true);
    plan->engine_m = m;
    plan->engine_f32 = f32;
    if (plan->engine->err != cudaSuccess) {
      const cudaError_t e = plan->engine->err;
      delete plan->engine;
      plan->engine = nullptr;
      return cuda_fail(e, what);
    }
  }
  Engine& E = *plan->engine;
  if (!job->setup(E.stream(), E.m(), E.f32())) return cuda_fail(cudaErrorMemoryAllocation, what);
  E.add(job);
  while (E.njobs() > 0) {
    if (!E.tick()) {
      const cudaError_t e = E.err;
      E.retire();
      delete plan->engine;
      plan->engine = nullptr;
      return cuda_fail(e, what);
    }
    for (Job* j : E.retire()) j->finish(E.stream());
  }
  const cudaError_t e = cudaStreamSynchronize(E.stream());
  if (e != cudaSuccess) return cuda_fail(e, what);
  return PI_OK;
}

void release_plan_engine(pi_plan* plan) {
  delete plan->engine;
  plan->engine = nullptr;
}

namespace {

int check_expv_opts(const pi_expv_opts_t* o) {
  if (!o) return fail(PI_ERR_INVALID_ARGUMENT, "null options");
  if (o->krylovdim < 1 || o->krylovdim > kBatchMaxKrylov)
    return fail(PI_ERR_INVALID_ARGUMENT, "krylovdim must lie in 1:120 for batched solves");
  if (!(o->atol >= 0) || !(o->rtol >= 0) || !std::isfinite(o->atol) || !std::isfinite(o->rtol))
    return fail(PI_ERR_INVALID_ARGUMENT, "atol and rtol must be finite nonnegative real numbers");
  if (!(o->safety > 0 && o->safety < 1))
    return fail(PI_ERR_INVALID_ARGUMENT, "safety must lie strictly between zero and one");
  if (o->max_steps < 1) return fail(PI_ERR_INVALID_ARGUMENT, "max_steps must be positive");
  if (o->precision != PI_FP64 && o->precision != PI_FP32)
    return fail(PI_ERR_INVALID_ARGUMENT, "precision must be PI_FP64 or PI_FP32");
  return PI_OK;
}

int check_gmres_opts(const pi_gmres_opts_t* o) {
  if (!o) return fail(PI_ERR_INVALID_ARGUMENT, "null options");
  if (o->krylovdim < 1 || o->krylovdim > kBatchMaxKrylov)
    return fail(PI_ERR_INVALID_ARGUMENT, "krylovdim must lie in 1:120 for batched solves");
  if (o->maxiter < 1) return fail(PI_ERR_INVALID_ARGUMENT, "maxiter must be positive");
  if (!(o->atol >= 0) || !(o->rtol >= 0)) return fail(PI_ERR_INVALID_ARGUMENT, "tolerances must be nonnegative");
  if (o->precision != PI_FP64 && o->precision != PI_FP32)
    return fail(PI_ERR_INVALID_ARGUMENT, "precision must be PI_FP64 or PI_FP32");
  if (o->preconditioner != nullptr || o->drive_preconditioner != nullptr || o->coords != PI_COORDS_REFERENCE)
    return fail(PI_ERR_UNSUPPORTED,
                "batched steady states run unpreconditioned in reference coordinates; solve preconditioned or "
                "population-coordinate steady states with pi_steady_state");
  return PI_OK;
}

int check_plans(int n, pi_plan* const* plans, double* const* states, int* device) {
  if (n < 1 || !plans || !states) return fail(PI_ERR_INVALID_ARGUMENT, "null argument");
  std::unordered_set<const void*> seen;
  for (int i = 0; i < n; ++i) {
    if (!plans[i] || !states[i]) return fail(PI_ERR_INVALID_ARGUMENT, "null plan or state in the batch");
    if (plans[i]->device != plans[0]->device)
      return fail(PI_ERR_INVALID_ARGUMENT, "all plans of a batch must live on one device");
    if (!seen.insert(states[i]).second)
      return fail(PI_ERR_INVALID_ARGUMENT, "two batch instances share one state buffer");
  }
  *device = plans[0]->device;
  return PI_OK;
}

// Runs the engine until every job finished; returns the first job error (or a CUDA error).
int run_jobs(Engine& E, std::vector<Job*>& jobs, const char* what) {
  for (Job* j : jobs) {
    if (!j->setup(E.stream(), E.m(), E.f32())) return cuda_fail(cudaErrorMemoryAllocation, what);
    E.add(j);
  }
  while (E.njobs() > 0) {
    if (!E.tick()) return cuda_fail(E.err, what);
    for (Job* j : E.retire()) j->finish(E.stream());
  }
  const cudaError_t e = cudaStreamSynchronize(E.stream());
  if (e != cudaSuccess) return cuda_fail(e, what);
  for (size_t i = 0; i < jobs.size(); ++i)
    if (jobs[i]->rc != PI_OK) {
      char m[64];
      std::snprintf(m, sizeof(m), "batch instance %zu: ", i);
      return fail(jobs[i]->rc, std::string(m) + jobs[i]->msg);
    }
  return PI_OK;
}

}  // namespace
}  // namespace picuda

using namespace picuda;

extern "C" {

int pi_expv_batch(int ninst, pi_plan* const* plans, double* const* x_devs, const double* t,
                  const pi_expv_opts_t* opts, pi_expv_info_t* infos) {
  int device = 0;
  int rc = check_plans(ninst, plans, x_devs, &device);
  if (rc) return rc;
  rc = check_expv_opts(opts);
  if (rc) return rc;
  if (!t) return fail(PI_ERR_INVALID_ARGUMENT, "null times");
  for (int i = 0; i < ninst; ++i)
    if (!std::isfinite(t[i])) return fail(PI_ERR_INVALID_ARGUMENT, "time must be finite");
  std::vector<DynamicsJob*> jobs;
  std::vector<Job*> base;
  for (int i = 0; i < ninst; ++i) {
    jobs.push_back(new DynamicsJob(plans[i], x_devs[i], {0.0, t[i]}, 0, nullptr, nullptr, *opts, true));
    base.push_back(jobs.back());
  }
  {
    Engine E(plans[0]->device, opts->krylovdim, opts->precision == PI_FP32, true);
    if (E.err != cudaSuccess) rc = cuda_fail(E.err, "batched expv engine");
    if (!rc) rc = run_jobs(E, base, "batched expv");
    if (infos)
      for (int i = 0; i < ninst; ++i) infos[i] = jobs[i]->info();
    for (Job* j : base) delete j;
  }
  (void)device;
  return rc;
}

int pi_dynamics_batch(int njobs, const pi_dynamics_job_t* specs, const pi_expv_opts_t* opts, pi_expv_info_t* infos) {
  if (njobs < 1 || !specs) return fail(PI_ERR_INVALID_ARGUMENT, "null argument");
  std::vector<pi_plan*> plans(njobs);
  std::vector<double*> states(njobs);
  for (int i = 0; i < njobs; ++i) {
    plans[i] = specs[i].plan;
    states[i] = specs[i].state_dev;
  }
  int device = 0;
  int rc = check_plans(njobs, plans.data(), states.data(), &device);
  if (rc) return rc;
  rc = check_expv_opts(opts);
  if (rc) return rc;
  for (int i = 0; i < njobs; ++i) {
    const pi_dynamics_job_t& s = specs[i];
    if (s.nt < 1 || !s.times) return fail(PI_ERR_INVALID_ARGUMENT, "every job needs at least one saved time");
    if (s.nobs < 0 || s.nobs > kBatchMaxObs || (s.nobs > 0 && (!s.obs_dev || !s.values_host)))
      return fail(PI_ERR_INVALID_ARGUMENT, "observables must number 0..16 with device data and a host output");
    for (int k = 0; k < s.nt; ++k) {
      if (!std::isfinite(s.times[k])) return fail(PI_ERR_INVALID_ARGUMENT, "saved times must be finite");
      if (k > 0 && !(s.times[k] >= s.times[k - 1]))
        return fail(PI_ERR_INVALID_ARGUMENT, "Krylov exponential output times must be nondecreasing");
    }
  }
  std::vector<DynamicsJob*> jobs;
  std::vector<Job*> base;
  for (int i = 0; i < njobs; ++i) {
    const pi_dynamics_job_t& s = specs[i];
    jobs.push_back(new DynamicsJob(s.plan, s.state_dev, std::vector<double>(s.times, s.times + s.nt), s.nobs,
                                   s.obs_dev, s.values_host, *opts, false));
    base.push_back(jobs.back());
  }
  {
    Engine E(device, opts->krylovdim, opts->precision == PI_FP32, true);
    if (E.err != cudaSuccess) rc = cuda_fail(E.err, "batched dynamics engine");
    if (!rc) rc = run_jobs(E, base, "batched dynamics");
    if (infos)
      for (int i = 0; i < njobs; ++i) infos[i] = jobs[i]->info();
    for (Job* j : base) delete j;
  }
  return rc;
}

int pi_engine_set_apply_schedule(int schedule) {
  if (schedule < PI_SCHEDULE_PER_TILE || schedule > 64)
    return fail(PI_ERR_INVALID_ARGUMENT, "schedule must be PI_SCHEDULE_AUTO, PI_SCHEDULE_PER_TILE or 1..64 blocks per SM");
  g_apply_schedule.store(schedule);
  return PI_OK;
}

int pi_engine_schedule_info(pi_schedule_info_t* out) {
  if (!out) return fail(PI_ERR_INVALID_ARGUMENT, "null output");
  std::lock_guard<std::mutex> lk(g_schedule_mu);
  *out = g_schedule_info;
  return PI_OK;
}

int pi_steady_state_batch(int ninst, pi_plan* const* plans, double* const* x_devs, const pi_gmres_opts_t* opts,
                          pi_gmres_info_t* infos) {
  int device = 0;
  int rc = check_plans(ninst, plans, x_devs, &device);
  if (rc) return rc;
  rc = check_gmres_opts(opts);
  if (rc) return rc;
  std::vector<SteadyJob*> jobs;
  std::vector<Job*> base;
  for (int i = 0; i < ninst; ++i) {
    jobs.push_back(new SteadyJob(plans[i], x_devs[i], *opts, 0x51ca1eULL));
    base.push_back(jobs.back());
  }
  {
    Engine E(device, opts->krylovdim, opts->precision == PI_FP32, true);
    if (E.err != cudaSuccess) rc = cuda_fail(E.err, "batched steady-state engine");
    if (!rc) rc = run_jobs(E, base, "batched steady state");
    if (infos)
      for (int i = 0; i < ninst; ++i) infos[i] = jobs[i]->info();
    for (Job* j : base) delete j;
  }
  return rc;
}

}  // extern "C"
