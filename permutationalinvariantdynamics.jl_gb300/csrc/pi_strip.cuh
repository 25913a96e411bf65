// Action of a canonical plan (real one-body qubit operators) from merged coefficient planes: one
// thread per output entry, entries of a sector block in memory order.
//
// What bounds it.  FP64: GB300 issues FP64 at 1/64 of its FP32 rate (a warp-wide FMA holds a
// quarter of an SM for 64 cycles), so the time is the number of FP64 instructions issued, those
// of padding lanes and of predicated-off lanes included.  FP32: the L1 wavefronts of the sources
// (three per misaligned 256-byte row of a warp).  Hence
//   - merged coefficients: every gain position keeps one precomputed coefficient per entry (one
//     plane per position and two for the centre), which leaves 4 (centre), 8 (line shifts) and 2
//     per gain position: 22 multiply-adds per entry with emission, dephasing and collective
//     decay, against 41 when every term's alpha[a] beta[b] is formed on the way;
//   - the gain positions of the plan are compile-time counted: a test in the kernel would be
//     if-converted and its FMAs issued all the same, and an absent position costs no load;
//   - lanes run over the flat entry index a + b n, so only the last warp of a sector block
//     has idle lanes; 32 x 32 tiles leave 20% of them idle at N = 120;
//   - sources are plain loads of one complex entry served by L1 and L2: no window has to be
//     staged before a block can start.
#pragma once

#include "pi_apply_impl.cuh"
#include "pi_device.cuh"

namespace picuda {

constexpr int kStripWarps = 4;  // items per block
constexpr int kStripThreads = 32 * kStripWarps;

// Kernel variants: gain slots and line shifts (drive).  A plan takes the first one that fits.
constexpr int kStripVariants = 7;
template <int V>
struct StripVariant {
  static constexpr int NR = V == 0 ? 1 : V == 1 ? 3 : V == 2 || V == 5 ? 5 : V == 3 ? 6 : 8;
  static constexpr bool H = V < 5;
};

// One thread's entry: where its sources are and the coefficients they take.  NC: the source
// vector is not written by the running kernel (loads through the read-only path).
template <typename T, int V, bool NC = true>
struct StripEntry {
  using T2 = typename Vec2<T>::type;
  static constexpr int NR = StripVariant<V>::NR;
  static constexpr bool H = StripVariant<V>::H;
  int e, n;      // element index, own dimension
  int at[NR];    // element index of each gain's source
  unsigned ok;   // sources inside their blocks: bits 0..NR-1 gains, 16.. row and column shifts
  bool diag;
  T cr, ci, c[NR];
  T2 l, r;

  // False for lanes past the sector block.
  __device__ __forceinline__ bool load(const StripItem& it, const StripPlanes<T>& P, int lane) {
    const int i = it.local0 + lane;
    n = it.n;
    if (i >= n * n) return false;
    const int b = (int)((unsigned)i / (unsigned)n), a = i - b * n;
    e = it.off + i;
    diag = a == b;
    const T* p = P.plane + e;
    cr = __ldg(p);
    ci = __ldg(p + P.dim);
    ok = 0;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const int src = P.gain[k].src;  // uniform
      const int m = src < 0 ? 0 : src == 0 ? n : src == 1 ? it.m0 : it.m2;
      const int off = src == 1 ? it.off0 : src == 2 ? it.off2 : it.off;
      const int d = P.gain[k].shift + (src == 1 ? -1 : src == 2 ? 1 : 0);
      const int u = a + d, v = b + d;
      // false for every u when the neighbour is missing (m = 0)
      const bool in = (unsigned)u < (unsigned)m && (unsigned)v < (unsigned)m;
      at[k] = off + u + v * m;
      c[k] = in ? __ldg(p + (2 + k) * P.dim) : T(0);
      ok |= in ? 1u << k : 0u;
    }
    if (H) {
      l = __ldg(P.lrow + it.loff + a);
      r = __ldg(P.rcol + it.loff + b);
      ok |= (a > 0 ? 1u << 16 : 0u) | (a < n - 1 ? 1u << 17 : 0u) | (b > 0 ? 1u << 18 : 0u) | (b < n - 1 ? 1u << 19 : 0u);
    }
    return true;
  }

  // (L x)[e].  Sources outside their block are zero and not read.
  __device__ __forceinline__ T2 apply(const T2* x) const {
    const T2* o = x + e;
    const T2 xc = ld(o);
    // all sources first: the loads are in flight together
    T2 g[NR], xu, xd, xl, xr;
    if (H) {
      xu = src(o - 1, 16);
      xd = src(o + 1, 17);
      xl = src(o - n, 18);
      xr = src(o + n, 19);
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) g[k] = src(x + at[k], k);
    T2 y;
    y.x = fma(-ci, xc.y, cr * xc.x);
    y.y = fma(ci, xc.x, cr * xc.y);
    if (H) {
      imag(y, l.x, xu);
      imag(y, l.y, xd);
      imag(y, r.x, xl);
      imag(y, r.y, xr);
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      y.x = fma(c[k], g[k].x, y.x);
      y.y = fma(c[k], g[k].y, y.y);
    }
    return y;
  }

 private:
  static __device__ __forceinline__ T2 ld(const T2* p) { return NC ? __ldg(p) : *p; }
  __device__ __forceinline__ T2 src(const T2* p, int k) const {
    return ok >> k & 1 ? ld(p) : T2{};
  }
  static __device__ __forceinline__ void imag(T2& y, T k, T2 v) {
    y.x = fma(-k, v.y, y.x);
    y.y = fma(k, v.x, y.y);
  }
};

}  // namespace picuda
