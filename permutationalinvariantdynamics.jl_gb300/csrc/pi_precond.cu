// Level-sweep preconditioner for the trace-fixed steady-state GMRES.
//
// The reference preconditions krylov_steady_state with the LU factors of the diagonal Schur
// blocks of L/s + v t^H (schur_sector_preconditioner, krylov.jl:183-700, applied on the left
// in _gmres!, krylov.jl:732-787).  That is one dense n^2 x n^2 factorisation per sector:
// O(n^6) work and a 40k x 40k matrix per sector at N = 200.  This file keeps the reference's
// left-preconditioned GMRES and replaces the factors by the exact inverse of a different
// part of L, one that a GPU can invert in O(dim) work.
//
// Write an entry of sector s as (a, b) with a = j - M and b = j - M' (GT order).  Every term
// of a qubit Liouvillian reads x_src[a + e + p, b + e + q].  The terms with p == q keep the
// charge d = b - a = M - M' (they commute with the U(1) rotation generated by Jz): the
// dissipators of Jz-covariant jump operators (sigma-, sigma+, sigma_z, J-, ...), the
// diagonal of the Hamiltonian, and the loss anticommutators.  The terms with p != q -- the
// drive, Jx and Jy -- change d by one.  L0, the charge-keeping part, is block diagonal in
// d.  Inside one charge block, with the level index lambda = 2M = n_s - 1 - 2a:
//   - p = q = 0 terms couple an entry to the same (M, M') in the sectors s-1, s, s+1:
//     a tridiagonal system over the sectors present at that level;
//   - p = q = -1 terms (decay-type gains) read the level lambda + 2, and p = q = +1 terms
//     (pump-type gains) read lambda - 2.
// When the gains all point one way, the block is block lower-triangular in lambda with
// tridiagonal diagonal blocks, so L0 z = r is solved exactly by sweeping the levels in that
// order with one Thomas solve per level.  The Thomas factors are computed once here.
//
// The bordered operator M = L0/s + v t^H is then inverted exactly, in one of two ways:
//   - L0 singular, its null vector on one "free" entry: the zero pivot of the last level of
//     the d = 0 chain (the all-down population for decay models).  Write z = y + c e_f with
//     beta = t^H z; then L0 y = s (r - beta v).  The sweep of s r with the free equation
//     dropped gives y_r and that equation's residual rho_r; the same for s v, precomputed,
//     gives y_v and rho_v.  The free equation fixes beta = rho_r / rho_v, so
//     y = y_r - beta y_v, and c = (beta - t^H y) / t_f.  (For a trace-preserving L0 this is
//     beta = t^H r.)
//   - L0 nonsingular (or regularised): Sherman-Morrison with the precomputed w0 = s L0^-1 v.
// v and t live on the block diagonals, which are exactly the d = 0 chain, and sweeps keep the
// charge, so y_v, w0 and both corrections stay inside the thread block that sweeps that
// chain.
//
// Device layout: one thread block per charge chain (2 n_max - 1 chains, the longest first).  The
// levels of a chain depend on one another, so the time is the latency of one level on the warp that
// solves it, and everything that does not depend on the previous level is taken off that warp.  A
// ring of shared-memory slots holds the levels at hand.  Each stager warp prepares every NS-th level
// alone: it copies the factors with cp.async, gathers r, replaces r by W s r, and forms the
// products of Thomas multipliers that the two scans combine with.  The solving warp takes a level
// when its slot is full, adds the gains of the previous level's solution (premultiplied by -W in
// the tables), runs both Thomas recurrences as warp-wide scans of affine maps (each lane composes a
// chunk of at most five entries; FP32 scans step by factors of four) and leaves the solution in
// the slot, from where the stager that takes the slot next writes it to z.  Full and done
// mbarriers order the warps; nothing waits for a whole block.  N = 200, FP32, per sweep of
// FP64 vectors: 235 us with block barriers and the store of z and the products on the solving
// warp, 161 us now; FP64 sweeps in reference coordinates 1188 us, now 822.  A level of 101 entries
// takes about 1300 cycles: gains 400, forward and backward scan 270 each, the rest waits and
// arrivals.  Loading the next level's entries into registers during the backward scan costs more
// (spills, or fewer stagers: 213 us).  Population coordinates run in FP32 (the preconditioner is an
// approximation of L^-1 either way, and every entry is a bounded population); reference coordinates
// run in FP64, since their entries span many decades at large N.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/picuda.h"
#include "pi_handle.hpp"
#include "pi_internal.hpp"
#include "pi_reduce.cuh"
#include "pi_precond.hpp"
#include "pi_drive.hpp"

namespace picuda {

namespace {

constexpr int kNoGain = 1023;

template <typename T>
struct V2;
template <>
struct V2<double> {
  using type = double2;
  static __host__ __device__ double2 make(double x, double y) { return make_double2(x, y); }
};
template <>
struct V2<float> {
  using type = float2;
  static __host__ __device__ float2 make(float x, float y) { return make_float2(x, y); }
};

template <typename T2>
__device__ __forceinline__ T2 cmul(T2 a, T2 b) {
  T2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
// c + a * b
template <typename T2>
__device__ __forceinline__ T2 cfma(T2 a, T2 b, T2 c) {
  T2 r;
  r.x = fma(a.x, b.x, fma(-a.y, b.y, c.x));
  r.y = fma(a.x, b.y, fma(a.y, b.x, c.y));
  return r;
}
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

template <typename TI>
__device__ __forceinline__ double2 load_d2(const TI* p) {
  const TI v = *p;
  return make_double2((double)v.x, (double)v.y);
}

template <typename TO, typename T2>
__device__ __forceinline__ void store_as(TO* p, T2 v);
template <>
__device__ __forceinline__ void store_as<double2, double2>(double2* p, double2 v) { *p = v; }
template <>
__device__ __forceinline__ void store_as<double2, float2>(double2* p, float2 v) {
  *p = make_double2((double)v.x, (double)v.y);
}
template <>
__device__ __forceinline__ void store_as<float2, float2>(float2* p, float2 v) { *p = v; }
template <>
__device__ __forceinline__ void store_as<float2, double2>(float2* p, double2 v) {
  *p = make_float2((float)v.x, (float)v.y);
}

// Block-wide sum of two doubles per thread (fixed order).
__device__ __forceinline__ double2 block_sum2(double2 v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, off);
    v.y += __shfl_down_sync(0xffffffffu, v.y, off);
  }
  __syncthreads();
  if (lane == 0) {
    red[2 * warp] = v.x;
    red[2 * warp + 1] = v.y;
  }
  __syncthreads();
  double2 out = make_double2(0.0, 0.0);
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    out.x += red[2 * w];
    out.y += red[2 * w + 1];
  }
  __syncthreads();
  return out;
}

static_assert(kPrecondMaxLevel <= 5 * 32, "the solving warp takes levels of at most five entries per lane");
// Stager warps, slots and scan coefficients per direction.  A stager has NS levels of time for one
// of its own, and starts it when the level SLOTS - 1 before it is solved.  A staged FP32 level costs
// several times the latency of a solved one (two dependent copies, then the products): N = 200
// takes 192 us with three stagers and six slots, 195 with four and five, 163 with four and six, 160
// with five and seven, 173 with seven and eight.  An FP64 level is bound by its sub-partition's FP64
// pipe on either side, and three stagers have a sub-partition each.  Both rings leave room for two
// blocks per SM.
template <typename T>
struct Ring;
template <>
struct Ring<float> {
  static constexpr int NS = 5, SLOTS = 7, COEFS = 7;
};
template <>
struct Ring<double> {
  static constexpr int NS = 3, SLOTS = 5, COEFS = 5;
};
template <typename T>
constexpr int kSweepThreads = 32 * (1 + Ring<T>::NS);
constexpr int kMaxChainLevels = 2 * kPrecondMaxLevel + 4;

__device__ __forceinline__ float2 shfl_up_c(float2 v, int d) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl_up_c(double2 v, int d) {
  return make_double2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ float2 shfl_down_c(float2 v, int d) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl_down_c(double2 v, int d) {
  return make_double2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}

__device__ __forceinline__ void cpa(void* smem, const void* gmem, int bytes) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(gmem) : "memory");
  else if (bytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(a), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(a), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Slot position of entry i of a level with K = ceil(cnt / 32) entries per lane: lane l's q-th
// entry (i = l K + q) sits at q * 32 + l, so the solving warp's accesses of one q are bank-conflict free.
__device__ __forceinline__ int slot_pos(int i, int K) { return (i % K) * 32 + i / K; }
__device__ __forceinline__ int level_width(int cnt) { return max((cnt + 31) >> 5, 1); }

// One staged level: its right-hand side, factors and gain tables.
template <typename T, typename TI>
struct Slot {
  using T2 = typename V2<T>::type;
  union {
    TI r[kPrecondMaxLevel];  // r at the level's elements, as stored
    T2 b[kPrecondMaxLevel];  // then W s r, then the solution
  };
  union {
    T2 w[kPrecondMaxLevel];           // 1 / pivot
    T2 pf[32 * Ring<T>::COEFS];       // then the forward scan's coefficients
  };
  T2 pb[32 * Ring<T>::COEFS];  // the backward scan's coefficients
  T2 a[kPrecondMaxLevel];      // forward multiplier
  T2 c[kPrecondMaxLevel];      // backward multiplier
  T2 g[3][kPrecondMaxLevel];   // gain coefficients times -W
  int gp[kPrecondMaxLevel];    // packed gain positions in the previous level
  int el[kPrecondMaxLevel];    // element index
};

template <typename T, typename TI>
struct SweepSmem {
  using T2 = typename V2<T>::type;
  static constexpr int kSlots = Ring<T>::SLOTS;
  Slot<T, TI> slot[kSlots];
  unsigned long long full[kSlots], done[kSlots];  // mbarriers
  double red[2 * (1 + Ring<T>::NS)];
  T2 none;                       // the first level's previous solution: a finite zero
  int lev_ent[kMaxChainLevels];  // the chain's level bounds
  int gave_up;
};

// One direction's affine maps compose from lane to lane as (P, Q)_l <- (P, Q)_l o (P, Q)_{l-D}
// (forward, UP) or l + D.  A step of N neighbours at distances D, 2D .. N D uses the coefficients
// out[j] = P_l P_{l-D} .. P_{l-jD}, zero where the neighbour does not exist; P becomes the product
// over the window of N + 1.
template <bool UP, int D, int N, typename T2>
__device__ __forceinline__ void coef_step(T2& P, T2* out, int lane) {
  const int room = UP ? lane : 31 - lane;  // lanes on the side that is read
  T2 c = P;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (j > 0) c = cmul(c, UP ? shfl_up_c(P, j * D) : shfl_down_c(P, j * D));
    T2 v = c;
    if (room < (j + 1) * D) v.x = v.y = 0;
    out[32 * j + lane] = v;
  }
  if (D * (N + 1) < 32) P = cmul(c, UP ? shfl_up_c(P, N * D) : shfl_down_c(P, N * D));
}
// The matching step on the constant parts.  A lane without that neighbour reads its own value and a
// zero coefficient.
template <bool UP, int D, int N, typename T2>
__device__ __forceinline__ void scan_step(T2& Q, const T2* coef, int lane) {
  T2 q[N];
#pragma unroll
  for (int j = 0; j < N; ++j) q[j] = UP ? shfl_up_c(Q, (j + 1) * D) : shfl_down_c(Q, (j + 1) * D);
#pragma unroll
  for (int j = 0; j < N; ++j) Q = cfma(coef[32 * j + lane], q[j], Q);
}
// FP32: two steps by four and one by two (latency counts); FP64: five steps by two (each FP64
// instruction of a warp holds the pipe for 64 cycles, so their number counts).
template <bool UP>
__device__ __forceinline__ void scan_coefs(float2 P, float2* out, int lane) {
  coef_step<UP, 1, 3>(P, out, lane);
  coef_step<UP, 4, 3>(P, out + 96, lane);
  coef_step<UP, 16, 1>(P, out + 192, lane);
}
template <bool UP>
__device__ __forceinline__ void scan(float2& Q, const float2* coef, int lane) {
  scan_step<UP, 1, 3>(Q, coef, lane);
  scan_step<UP, 4, 3>(Q, coef + 96, lane);
  scan_step<UP, 16, 1>(Q, coef + 192, lane);
}
template <bool UP>
__device__ __forceinline__ void scan_coefs(double2 P, double2* out, int lane) {
  coef_step<UP, 1, 1>(P, out, lane);
  coef_step<UP, 2, 1>(P, out + 32, lane);
  coef_step<UP, 4, 1>(P, out + 64, lane);
  coef_step<UP, 8, 1>(P, out + 96, lane);
  coef_step<UP, 16, 1>(P, out + 128, lane);
}
template <bool UP>
__device__ __forceinline__ void scan(double2& Q, const double2* coef, int lane) {
  scan_step<UP, 1, 1>(Q, coef, lane);
  scan_step<UP, 2, 1>(Q, coef + 32, lane);
  scan_step<UP, 4, 1>(Q, coef + 64, lane);
  scan_step<UP, 8, 1>(Q, coef + 96, lane);
  scan_step<UP, 16, 1>(Q, coef + 128, lane);
}

// One stager warp prepares a level of cnt entries from e0 in slot L; entries past the level up to
// the K-th of lane 31 become zeros, so that the solving warp needs no bounds.
template <typename T, typename TI>
__device__ __forceinline__ void stage_level(const PrecondDev& P, Slot<T, TI>& L, const TI* __restrict__ r, int e0,
                                            int cnt, T s, int lane) {
  using T2 = typename V2<T>::type;
  const T2* W = reinterpret_cast<const T2*>(P.W);
  const T2* A = reinterpret_cast<const T2*>(P.A);
  const T2* C = reinterpret_cast<const T2*>(P.C);
  const T2* G = reinterpret_cast<const T2*>(P.G);
  const T2 zero = V2<T>::make((T)0, (T)0);
  const int K = level_width(cnt);
  for (int i = lane; i < 32 * K; i += 32) {
    const int p = slot_pos(i, K), e = e0 + i;
    if (i < cnt) {
      cpa(&L.el[p], P.elem + e, 4);
      cpa(&L.gp[p], P.gsrc + e, 4);
      cpa(&L.w[p], W + e, sizeof(T2));
      cpa(&L.a[p], A + e, sizeof(T2));
      cpa(&L.c[p], C + e, sizeof(T2));
#pragma unroll
      for (int q = 0; q < 3; ++q) cpa(&L.g[q][p], G + 3LL * e + q, sizeof(T2));
    } else {
      L.gp[p] = 0;
      L.w[p] = L.a[p] = L.c[p] = L.g[0][p] = L.g[1][p] = L.g[2][p] = zero;
    }
  }
  cpa_commit();
  cpa_wait<0>();
  for (int i = lane; i < cnt; i += 32) {  // the elements whose indices this lane copied
    const int p = slot_pos(i, K);
    cpa(&L.r[p], r + L.el[p], sizeof(TI));
  }
  cpa_commit();
  // meanwhile the chunk products; A and C of a lane were copied by others
  __syncwarp();
  T2 PA = L.a[lane], PC = L.c[lane];
  for (int q = 1; q < K; ++q) {
    PA = cmul(PA, L.a[q * 32 + lane]);
    PC = cmul(PC, L.c[q * 32 + lane]);
  }
  scan_coefs<false>(PC, L.pb, lane);
  cpa_wait<0>();
  __syncwarp();
  // W s r in place: all of r and W is read before the first write
  T2 v[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    if (q >= K) break;
    const int p = q * 32 + lane, i = lane * K + q;
    if (i < cnt) {
      const TI x = L.r[p];
      v[q] = V2<T>::make(s * (T)x.x, s * (T)x.y);
      if (e0 + i != P.free_ent) v[q] = cmul(L.w[p], v[q]);  // the free entry keeps s r for its residual
    } else {
      v[q] = zero;
    }
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 5; ++q)
    if (q < K) L.b[q * 32 + lane] = v[q];
  scan_coefs<true>(PA, L.pf, lane);
}

// t^H z over a thread's entries: FP64 with the weights t, or, in population coordinates, where t is
// one, of FP32 values (or double-floats) in triple-float.
struct TraceSum64 {
  double2 s = make_double2(0.0, 0.0);
  __device__ __forceinline__ void add(const PrecondDev& P, int e, double2 u) {
    const double t = P.t0[e - P.chain0_ent];
    s.x = fma(t, u.x, s.x);
    s.y = fma(t, u.y, s.y);
  }
  __device__ __forceinline__ double2 value() const { return s; }
};
struct TraceSumTF {
  TF x{0.f, 0.f, 0.f}, y{0.f, 0.f, 0.f};
  __device__ __forceinline__ void add(const PrecondDev&, int, float2 u) {
    tf_add(x, u.x);
    tf_add(y, u.y);
  }
  __device__ __forceinline__ void add(DF u, DF v) {
    tf_add(x, u.hi);
    tf_add(x, u.lo);
    tf_add(y, v.hi);
    tf_add(y, v.lo);
  }
  __device__ __forceinline__ double2 value() const { return make_double2(tf_value(x), tf_value(y)); }
};

// The solution of a level goes from its slot to z, and into the sum t^H z where that is wanted.
template <typename T, typename TI, typename TO, typename Sum>
__device__ __forceinline__ void drain_level(const PrecondDev& P, const Slot<T, TI>& L, TO* __restrict__ z, int e0,
                                            int cnt, bool sum_t, int lane, Sum& sum) {
  const int K = level_width(cnt);
  for (int i = lane; i < cnt; i += 32) {
    const int p = slot_pos(i, K);
    store_as<TO, typename V2<T>::type>(z + L.el[p], L.b[p]);
    if (sum_t) sum.add(P, e0 + i, L.b[p]);
  }
}

// ---- mbarriers with bounded waits
constexpr int kSweepWaitLimit = 1 << 20;  // polls, each of about a microsecond at most

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
// Waits for the phase with the given parity to complete; false after kSweepWaitLimit polls.
__device__ __forceinline__ bool bar_wait(unsigned long long* b, unsigned parity) {
  for (int it = 0; it < kSweepWaitLimit; ++it) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(b)), "r"(parity), "r"(1000)  // ns
        : "memory");
    if (done) return true;
  }
  return false;
}

// The solve of one staged level, K = ceil(cnt / 32) entries per lane.  Lane l owns the K
// consecutive entries l K .. l K + K - 1 (positions q 32 + l).  Right-hand sides b_i = W_i (s r_i
// - gains of the previous level's solution); the lane that meets the free entry keeps its unscaled
// residual.  Both Thomas recurrences, y_i = A_i y_{i-1} + b_i and u_i = C_i u_{i+1} + y_i, are
// affine maps composed over each lane's chunk, combined across lanes by a scan, then
// replayed inside the chunk.  Specialised on K so that short levels issue short code.
template <typename T, typename TI, int K>
__device__ __forceinline__ void solve_level(const PrecondDev& Pd, Slot<T, TI>& L, const typename V2<T>::type* uprev,
                                            int e0, int cnt, int lane, double2& rho_r, bool& has_rho) {
  using T2 = typename V2<T>::type;
  const T2 zero = V2<T>::make((T)0, (T)0);
  // the chunk index of the free entry; a level's padding has the next level's entry numbers
  const int free_q = Pd.free_ent - e0 < cnt ? Pd.free_ent - e0 - lane * K : -1;
  T2 B[K], A[K], C[K];
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int p = q * 32 + lane;
    const int packed = L.gp[p];  // an absent gain reads entry 0 with a zero coefficient
    T2 b = cfma(L.g[0][p], uprev[packed & 1023], L.b[p]);
    b = cfma(L.g[1][p], uprev[(packed >> 10) & 1023], b);
    B[q] = cfma(L.g[2][p], uprev[packed >> 20], b);
    A[q] = L.a[p];
    C[q] = L.c[p];
    if (q == free_q) {
      rho_r = make_double2((double)B[q].x, (double)B[q].y);
      has_rho = true;
      B[q] = zero;
    }
  }
  T2 Q = B[0];
#pragma unroll
  for (int q = 1; q < K; ++q) Q = cfma(A[q], Q, B[q]);
  scan<true>(Q, L.pf, lane);
  T2 y = shfl_up_c(Q, 1);
  if (lane == 0) y = zero;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    y = cfma(A[q], y, B[q]);
    B[q] = y;
  }
  Q = B[K - 1];
#pragma unroll
  for (int q = K - 2; q >= 0; --q) Q = cfma(C[q], Q, B[q]);
  scan<false>(Q, L.pb, lane);
  T2 u = shfl_down_c(Q, 1);
  if (lane == 31) u = zero;
#pragma unroll
  for (int q = K - 1; q >= 0; --q) {
    u = cfma(C[q], u, B[q]);
    L.b[q * 32 + lane] = u;
  }
}

// The d = 0 chain's correction z -= k w0 at entries c0 .. c1.  One block does it for the whole
// chain (10,201 entries at N = 200), so eight entries per thread are in flight together: one by
// one, their two dependent gathers took a third of the sweep.  Returns the thread's share of t^H z,
// summed over the corrected values before they are rounded to TO: the free entry balances the trace
// of what was stored, and t^H y_r - k t^H w0 from sums of its own is off by the roundings of
// two large sums (N = 61..128 in FP64: 2e-14 of sum t |z|, against 2e-16).
constexpr int kTailUnroll = 8;

template <bool POP, typename TO>  // POP: population coordinates, where t is one
__device__ __forceinline__ double2 chain0_correct(const PrecondDev& Pd, TO* z, int c0, int c1, double2 k) {
  double2 sum = make_double2(0.0, 0.0);
  for (int e0 = c0 + threadIdx.x; e0 < c1; e0 += kTailUnroll * blockDim.x) {
    int el[kTailUnroll];
    double2 w[kTailUnroll], v[kTailUnroll];
    double t[kTailUnroll];
#pragma unroll
    for (int q = 0; q < kTailUnroll; ++q) {
      const int e = e0 + q * blockDim.x;
      el[q] = e < c1 ? Pd.elem[e] : -1;
      w[q] = e < c1 ? Pd.w0[e - c0] : make_double2(0.0, 0.0);
      t[q] = !POP && e < c1 ? Pd.t0[e - c0] : 1.0;
    }
#pragma unroll
    for (int q = 0; q < kTailUnroll; ++q) v[q] = el[q] >= 0 ? load_d2(z + el[q]) : make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < kTailUnroll; ++q) {
      if (el[q] < 0) continue;
      v[q].x = fma(-k.x, w[q].x, fma(k.y, w[q].y, v[q].x));
      v[q].y = fma(-k.x, w[q].y, fma(-k.y, w[q].x, v[q].y));
      store_as<TO, double2>(z + el[q], v[q]);
      sum.x = POP ? sum.x + v[q].x : fma(t[q], v[q].x, sum.x);
      sum.y = POP ? sum.y + v[q].y : fma(t[q], v[q].y, sum.y);
    }
  }
  return sum;
}

// The same for FP32 vectors: in double-float, as each conversion and FP64 operation of a warp
// holds a quarter of the SM's FP64 pipe for 64 cycles.
__device__ __forceinline__ double2 chain0_correct_df(const PrecondDev& Pd, float2* z, int c0, int c1, double2 k) {
  TraceSumTF sum;
  const DF kx{(float)k.x, (float)(k.x - (double)(float)k.x)}, ky{(float)k.y, (float)(k.y - (double)(float)k.y)};
  for (int e0 = c0 + threadIdx.x; e0 < c1; e0 += kTailUnroll * blockDim.x) {
    int el[kTailUnroll];
    float4 w[kTailUnroll];
    float2 v[kTailUnroll];
#pragma unroll
    for (int q = 0; q < kTailUnroll; ++q) {
      const int e = e0 + q * blockDim.x;
      el[q] = e < c1 ? Pd.elem[e] : -1;
      w[q] = e < c1 ? Pd.w0f[e - c0] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < kTailUnroll; ++q) v[q] = el[q] >= 0 ? z[el[q]] : make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < kTailUnroll; ++q) {
      if (el[q] < 0) continue;
      // w = (x.hi, x.lo, y.hi, y.lo)
      DF zx{v[q].x, 0.f}, zy{v[q].y, 0.f};
      df_axpy(zx, -kx.hi, -kx.lo, w[q].x);
      df_axpy(zx, ky.hi, ky.lo, w[q].z);
      zx.lo = fmaf(-kx.hi, w[q].y, fmaf(ky.hi, w[q].w, zx.lo));
      df_axpy(zy, -kx.hi, -kx.lo, w[q].z);
      df_axpy(zy, -ky.hi, -ky.lo, w[q].x);
      zy.lo = fmaf(-kx.hi, w[q].w, fmaf(-ky.hi, w[q].y, zy.lo));
      z[el[q]] = make_float2(zx.hi + zx.lo, zy.hi + zy.lo);
      sum.add(zx, zy);
    }
  }
  return sum.value();
}

template <typename T, typename TI, typename TO>
__global__ void __launch_bounds__(kSweepThreads<T>, 2)
    k_level_sweep(const PrecondDev Pd, const TI* __restrict__ r, TO* __restrict__ z, double s) {
  using T2 = typename V2<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepSmem<T, TI>& S = *reinterpret_cast<SweepSmem<T, TI>*>(smem_raw);
  const int chain = Pd.chain_order[blockIdx.x];
  const int lev0 = Pd.chain_lev[chain], lev1 = Pd.chain_lev[chain + 1];
  const int nlev = lev1 - lev0;
  const bool chain0 = chain == Pd.chain0;
  const bool sum_t = chain0 && Pd.mode == 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kSlots = Ring<T>::SLOTS, NS = Ring<T>::NS;
  for (int k = tid; k <= nlev; k += blockDim.x) S.lev_ent[k] = Pd.lev_ent[lev0 + k];
  if (tid < kSlots) {
    bar_init(&S.full[tid], 1);
    bar_init(&S.done[tid], 1);
  }
  if (tid == 0) {
    S.none = V2<T>::make((T)0, (T)0);
    S.gave_up = 0;
  }
  __syncthreads();
  double2 tsum = make_double2(0.0, 0.0);
  double2 rho_r = make_double2(0.0, 0.0);  // residual of the dropped free equation (lane-held)
  bool has_rho = false;
  if (warp > 0) {
    const T sT = (T)s;
    typename std::conditional<std::is_same<T, float>::value, TraceSumTF, TraceSum64>::type sum;
    for (int k = warp - 1; k < nlev + kSlots; k += NS) {
      // level k takes the slot of level k - kSlots, whose solution level k - kSlots + 1 has read
      const int out = k - kSlots;
      if (out >= 0) {
        const int by = min(out + 1, nlev - 1);
        if (!bar_wait(&S.done[by % kSlots], (unsigned)(by / kSlots) & 1u)) {
          S.gave_up = 1;
          break;
        }
        const int e0 = S.lev_ent[out], cnt = S.lev_ent[out + 1] - e0;
        drain_level<T, TI, TO>(Pd, S.slot[out % kSlots], z, e0, cnt, sum_t, lane, sum);
        __syncwarp();
      }
      if (k < nlev) {
        stage_level<T, TI>(Pd, S.slot[k % kSlots], r, S.lev_ent[k], S.lev_ent[k + 1] - S.lev_ent[k], sT, lane);
        __syncwarp();
        if (lane == 0) bar_arrive(&S.full[k % kSlots]);
      }
    }
    tsum = sum.value();
  } else {
    const T2* up = &S.none;
    for (int k = 0; k < nlev; ++k) {
      const int e0 = S.lev_ent[k], cnt = S.lev_ent[k + 1] - e0;
      if (!bar_wait(&S.full[k % kSlots], (unsigned)(k / kSlots) & 1u)) {
        S.gave_up = 1;
        break;
      }
      Slot<T, TI>& L = S.slot[k % kSlots];
      switch (level_width(cnt)) {
        case 1: solve_level<T, TI, 1>(Pd, L, up, e0, cnt, lane, rho_r, has_rho); break;
        case 2: solve_level<T, TI, 2>(Pd, L, up, e0, cnt, lane, rho_r, has_rho); break;
        case 3: solve_level<T, TI, 3>(Pd, L, up, e0, cnt, lane, rho_r, has_rho); break;
        case 4: solve_level<T, TI, 4>(Pd, L, up, e0, cnt, lane, rho_r, has_rho); break;
        default: solve_level<T, TI, 5>(Pd, L, up, e0, cnt, lane, rho_r, has_rho); break;
      }
      up = L.b;
      __syncwarp();  // the level's solution is in place for every lane
      if (lane == 0) bar_arrive(&S.done[k % kSlots]);
    }
  }
  __syncthreads();
  if (S.gave_up) {  // a wait ran out: leave no number behind
    if (tid == 0)
      store_as<TO, double2>(z + Pd.elem[Pd.lev_ent[lev0]], make_double2(nan(""), nan("")));
    return;
  }
  if (!chain0) return;
  const int c0 = Pd.chain0_ent, c1 = Pd.lev_ent[lev1];
  double2 k;
  if (Pd.mode == 0) {
    // beta = rho_r / rho_v; y = y_r - beta y_v; z_f = (beta - t^H y) / t_f
    if (has_rho) {  // one lane
      const double2 iv = Pd.sm_coef;  // 1 / rho_v
      S.red[0] = rho_r.x * iv.x - rho_r.y * iv.y;
      S.red[1] = rho_r.x * iv.y + rho_r.y * iv.x;
    }
    __syncthreads();
    k = make_double2(S.red[0], S.red[1]);
    __syncthreads();  // red is free
  } else {
    // Sherman-Morrison: z -= w0 (t^H y) / (1 + t^H w0)
    const double2 tz = block_sum2(tsum, S.red);
    k = make_double2(tz.x * Pd.sm_coef.x - tz.y * Pd.sm_coef.y, tz.x * Pd.sm_coef.y + tz.y * Pd.sm_coef.x);
  }
  double2 share;
  if constexpr (std::is_same<T, float>::value && std::is_same<TO, float2>::value)
    share = chain0_correct_df(Pd, z, c0, c1, k);
  else
    share = chain0_correct<std::is_same<T, float>::value>(Pd, z, c0, c1, k);
  if (Pd.mode != 0) return;
  const double2 tz = block_sum2(share, S.red);  // of every entry but the free one, which is zero so far
  if (tid == 0 && Pd.free_ent >= 0)
    store_as<TO, double2>(z + Pd.elem[Pd.free_ent],
                          make_double2((k.x - tz.x) / Pd.free_t, (k.y - tz.y) / Pd.free_t));
}

template <typename T, typename TI, typename TO>
cudaError_t launch_sweep(const PrecondDev& D, int blocks, const void* r, void* z, double scale, cudaStream_t stream) {
  const size_t smem = sizeof(SweepSmem<T, TI>);
  // the shared-memory opt-in is a per-function, per-device attribute: set once per device
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ULL << (dev & 63);
  if (!(configured.load() & bit)) {
    e = cudaFuncSetAttribute(k_level_sweep<T, TI, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit);
  }
  k_level_sweep<T, TI, TO><<<blocks, kSweepThreads<T>, smem, stream>>>(D, (const TI*)r, (TO*)z, scale);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// Host construction
// ---------------------------------------------------------------------------------------

using cdv = std::complex<double>;

cdv term_coef(const StencilTerm& t, int a, int b) {
  switch (t.kind) {
    case ST_ADD: return t.alpha[a] + t.beta[b];
    case ST_LEFT: return t.alpha[a];
    case ST_RIGHT: return t.beta[b];
    default: return t.alpha[a] * t.beta[b];
  }
}

}  // namespace

int build_level_precond(const QubitPlan& hp, int coords, double regularization, double scale, LevelPrecondHost* out,
                        std::string* err) {
  LevelPrecondHost& H = *out;
  H = LevelPrecondHost{};
  const int S = (int)hp.sectors.size();
  if (S < 1) {
    *err = "empty basis";
    return PI_ERR_INVALID_ARGUMENT;
  }
  if (S > kPrecondMaxLevel) {
    *err = "the level-sweep preconditioner supports at most 160 sectors (N <= 318)";
    return PI_ERR_UNSUPPORTED;
  }
  if (hp.dim > 0x7fffffffLL) {
    *err = "basis too large for 32-bit element indices";
    return PI_ERR_UNSUPPORTED;
  }
  H.coords = coords;
  H.scale = scale;
  H.regularization = regularization;
  // classify the terms of every sector
  struct Lists {
    std::vector<const StencilTerm*> diag, side, gain;
  };
  std::vector<Lists> L(S);
  int dir = 0;  // -1: gains read level lambda + 2 (sweep lambda downward); +1 the reverse
  for (int s = 0; s < S; ++s) {
    for (const StencilTerm& t : hp.sectors[s].terms) {
      if (t.p != t.q) continue;  // changes the charge d: the drive, left out of L0
      if (t.p == 0) {
        if (t.src == s && t.e == 0) {
          L[s].diag.push_back(&t);
        } else if (t.src == s - 1 || t.src == s + 1) {
          L[s].side.push_back(&t);
        } else {
          *err = "a charge-keeping term couples non-adjacent sectors";
          return PI_ERR_UNSUPPORTED;
        }
      } else if (t.p == -1 || t.p == 1) {
        if (t.src < s - 1 || t.src > s + 1) {
          *err = "a charge-keeping gain couples non-adjacent sectors";
          return PI_ERR_UNSUPPORTED;
        }
        const int d = t.p < 0 ? -1 : 1;
        if (dir != 0 && dir != d) {
          *err = "the level-sweep preconditioner needs all charge-keeping gains to raise, or all to lower, the "
                 "magnetic number (decay-type or pump-type channels, not both)";
          return PI_ERR_UNSUPPORTED;
        }
        dir = d;
        L[s].gain.push_back(&t);
      } else {
        *err = "a charge-keeping term reaches more than one level";
        return PI_ERR_UNSUPPORTED;
      }
    }
  }
  if (dir == 0) dir = -1;
  H.direction = dir;
  std::vector<int> n(S);
  std::vector<double> sqf(S), f(S);
  for (int s = 0; s < S; ++s) {
    n[s] = hp.sectors[s].n;
    sqf[s] = hp.sectors[s].sqrt_f;
    f[s] = hp.sectors[s].f;
  }
  auto ratio = [&](int s, int src) { return coords == PI_COORDS_POPULATION ? sqf[s] / sqf[src] : 1.0; };
  const int nmax = n[0];
  // levels lambda = n - 1 - 2a, all of the parity of nmax - 1
  std::vector<int> lams;
  for (int lam = nmax - 1; lam >= -(nmax - 1); lam -= 2) lams.push_back(lam);
  if (dir > 0) std::reverse(lams.begin(), lams.end());
  // chains d = -(nmax-1) .. nmax-1
  double maxdiag = 0.0;
  std::vector<int> chain_len;
  H.chain_lev.push_back(0);
  H.lev_ent.push_back(0);
  for (int d = -(nmax - 1); d <= nmax - 1; ++d) {
    if (d == 0) H.chain0 = (int)H.chain_lev.size() - 1;
    const int chain_first_entry = (int)H.elem.size();
    for (int lam : lams) {
      const int need = std::max(std::abs(lam), std::abs(lam - 2 * d));
      int cnt = 0;
      while (cnt < S && n[cnt] - 1 >= need) ++cnt;
      if (cnt == 0) continue;
      if (d == 0 && H.chain0_ent < 0) H.chain0_ent = (int)H.elem.size();
      // tridiagonal coefficients over the sectors 0..cnt-1 at this (d, lambda)
      std::vector<cdv> D(cnt), lo(cnt), up(cnt);
      std::vector<double> mag(cnt, 0.0);
      for (int s = 0; s < cnt; ++s) {
        const int a = (n[s] - 1 - lam) / 2, b = a + d;
        H.elem.push_back((int)(hp.sectors[s].offset + a + (long long)b * n[s]));
        cdv dv = 0.0;
        for (const StencilTerm* t : L[s].diag) {
          const cdv c = term_coef(*t, a, b);
          dv += c;
          mag[s] += std::abs(c);
        }
        if (regularization > 0) dv += regularization * scale;
        D[s] = dv;
        for (const StencilTerm* t : L[s].side) {
          const int src = t->src;
          const int as = a + t->e, bs = b + t->e;
          if (as < 0 || bs < 0 || as >= n[src] || bs >= n[src] || src >= cnt) continue;
          const cdv c = term_coef(*t, a, b) * ratio(s, src);
          if (src == s - 1)
            lo[s] += c;
          else
            up[s] += c;
        }
        // gains from the previous level
        cdv g[3] = {0.0, 0.0, 0.0};
        bool has[3] = {false, false, false};
        for (const StencilTerm* t : L[s].gain) {
          const int src = t->src;
          const int as = a + t->e + t->p, bs = b + t->e + t->q;
          if (as < 0 || bs < 0 || as >= n[src] || bs >= n[src]) continue;
          const int slot = src - s + 1;
          g[slot] += term_coef(*t, a, b) * ratio(s, src);
          has[slot] = true;
        }
        int packed = 0;
        for (int k = 0; k < 3; ++k) {
          const int pos = has[k] ? s + k - 1 : kNoGain;
          packed |= pos << (10 * k);
          H.G.push_back(has[k] ? g[k] : cdv(0.0));
        }
        H.gsrc.push_back(packed);
        maxdiag = std::max(maxdiag, std::abs(dv));
      }
      // Thomas factors
      cdv cprev = 0.0;
      for (int s = 0; s < cnt; ++s) {
        const cdv lc = s > 0 ? lo[s] * cprev : cdv(0.0);
        const cdv piv = D[s] - lc;
        const double tol = 1e-11 * (mag[s] + std::abs(lc) + std::abs(D[s]));
        const long long e = (long long)H.elem.size() - cnt + s;
        if (std::abs(piv) <= tol || piv == cdv(0.0)) {
          H.zero_pivots.push_back(e);
          H.W.push_back(0.0);
          H.A.push_back(0.0);
          H.C.push_back(0.0);
          cprev = 0.0;
          continue;
        }
        const cdv w = 1.0 / piv;
        H.W.push_back(w);
        H.A.push_back(s > 0 ? -lo[s] * w : cdv(0.0));
        cprev = up[s] * w;
        H.C.push_back(-cprev);
      }
      H.lev_ent.push_back((int)H.elem.size());
      H.max_level = std::max(H.max_level, cnt);
    }
    H.chain_lev.push_back((int)H.lev_ent.size() - 1);
    chain_len.push_back((int)H.elem.size() - chain_first_entry);
  }
  H.maxdiag = maxdiag;
  for (size_t c = 0; c + 1 < H.chain_lev.size(); ++c)
    if (H.chain_lev[c + 1] - H.chain_lev[c] > 2 * kPrecondMaxLevel + 2) {
      *err = "a charge chain has more levels than the sweep kernel stages";
      return PI_ERR_UNSUPPORTED;
    }
  if ((long long)H.elem.size() != hp.dim) {
    *err = "level decomposition does not cover the basis";
    return PI_ERR_UNSUPPORTED;
  }
  // chain 0 data: trace weights t and border v (in the solve's coordinates)
  const int c0 = H.chain0;
  const int e0 = H.chain0_ent, e1 = H.lev_ent[H.chain_lev[c0 + 1]];
  for (int e = e0; e < e1; ++e) {
    const long long el = H.elem[e];
    int s = S - 1;
    while (s > 0 && hp.sectors[s].offset > el) --s;
    const double t = coords == PI_COORDS_POPULATION ? 1.0 : sqf[s];
    const double v = coords == PI_COORDS_POPULATION ? f[s] / hp.trace_norm2 : sqf[s] / hp.trace_norm2;
    H.t0.push_back(t);
    H.v0.push_back(v);
  }
  // the free entry: one zero pivot, alone in the last level of the d = 0 chain
  const int last_lev = H.chain_lev[c0 + 1] - 1;
  const bool last_single = H.lev_ent[last_lev + 1] - H.lev_ent[last_lev] == 1;
  if (H.zero_pivots.size() == 1 && H.zero_pivots[0] == e1 - 1 && last_single) {
    H.mode = 0;
    H.free_ent = (int)H.zero_pivots[0];
  } else if (!H.zero_pivots.empty()) {
    *err = "a level block of the preconditioner is singular; pass a small regularization";
    return PI_ERR_INVALID_ARGUMENT;
  } else {
    H.mode = 1;
  }
  // Host sweep of s v over the d = 0 chain in FP64 (the free equation dropped): y_v, and
  // rho_v, the dropped equation's residual (mode 0), or w0 = s L0^-1 v (mode 1).
  {
    const int nl0 = H.chain_lev[c0], nl1 = H.chain_lev[c0 + 1];
    std::vector<cdv> yv(e1 - e0, 0.0);
    std::vector<cdv> prevu, curu;
    cdv rho_v = 0.0;
    for (int lev = nl0; lev < nl1; ++lev) {
      const int b0 = H.lev_ent[lev], cnt = H.lev_ent[lev + 1] - b0;
      std::vector<cdv> y(cnt);
      for (int i = 0; i < cnt; ++i) {
        const int e = b0 + i;
        cdv rv = scale * H.v0[e - e0];
        for (int k = 0; k < 3; ++k) {
          const int pos = (H.gsrc[e] >> (10 * k)) & 1023;
          if (pos != kNoGain) rv -= H.G[3LL * e + k] * prevu[pos];
        }
        if (e == H.free_ent) rho_v = rv;
        y[i] = H.W[e] * rv;
        if (i > 0) y[i] += H.A[e] * y[i - 1];
      }
      curu.assign(cnt, 0.0);
      for (int i = cnt - 1; i >= 0; --i) curu[i] = y[i] + (i + 1 < cnt ? H.C[b0 + i] * curu[i + 1] : cdv(0.0));
      for (int i = 0; i < cnt; ++i) yv[b0 + i - e0] = curu[i];
      prevu = curu;
    }
    H.w0 = yv;
    if (H.mode == 0) {
      if (std::abs(rho_v) == 0.0) {
        *err = "the trace border does not fix the free entry of the preconditioner; pass a small regularization";
        return PI_ERR_INVALID_ARGUMENT;
      }
      H.sm_coef = rho_v;
    } else {
      cdv tw = 0.0;
      for (int e = e0; e < e1; ++e) tw += H.t0[e - e0] * yv[e - e0];
      H.sm_coef = 1.0 / (1.0 + tw);
    }
  }
  // schedule: longest chains first
  H.chain_order.resize(chain_len.size());
  for (size_t i = 0; i < chain_len.size(); ++i) H.chain_order[i] = (int)i;
  std::stable_sort(H.chain_order.begin(), H.chain_order.end(),
                   [&](int x, int y) { return chain_len[x] > chain_len[y]; });
  return PI_OK;
}

}  // namespace picuda

struct pi_precond {
  pi_plan* plan = nullptr;
  int kind = PI_PRECOND_LEVEL;
  picuda::LevelPrecondHost host;  // kind LEVEL: the tables; both kinds: coords and scale
  picuda::PrecondDev dev{};
  picuda::DriveState* drive = nullptr;  // kind DRIVE
  int fp64 = 0;
  size_t bytes = 0;
  double setup_seconds = 0.0;
  std::vector<void*> allocs;
};

namespace picuda {
namespace {

template <typename X>
int upload_vec(pi_precond* P, const std::vector<X>& v, const X** out) {
  void* p = nullptr;
  const size_t bytes = std::max<size_t>(sizeof(X) * v.size(), 16);
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) return cuda_fail(e, "preconditioner tables");
  P->allocs.push_back(p);
  P->bytes += bytes;
  if (!v.empty()) {
    e = cudaMemcpy(p, v.data(), sizeof(X) * v.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "preconditioner upload");
  }
  *out = (const X*)p;
  return PI_OK;
}

template <typename T>
int upload_factors(pi_precond* P) {
  using T2 = typename V2<T>::type;
  const LevelPrecondHost& H = P->host;
  auto conv = [](const std::vector<cdv>& v) {
    std::vector<T2> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) o[i] = V2<T>::make((T)v[i].real(), (T)v[i].imag());
    return o;
  };
  int rc;
  const T2* p = nullptr;
  if ((rc = upload_vec(P, conv(H.W), &p))) return rc;
  P->dev.W = p;
  if ((rc = upload_vec(P, conv(H.A), &p))) return rc;
  P->dev.A = p;
  if ((rc = upload_vec(P, conv(H.C), &p))) return rc;
  P->dev.C = p;
  // the gains times -W; the free entry (W = 0) keeps -G for its residual
  std::vector<cdv> G(H.G.size());
  for (size_t e = 0; e < H.W.size(); ++e)
    for (int q = 0; q < 3; ++q)
      G[3 * e + q] = (long long)e == H.free_ent ? -H.G[3 * e + q] : -H.W[e] * H.G[3 * e + q];
  if ((rc = upload_vec(P, conv(G), &p))) return rc;
  P->dev.G = p;
  return PI_OK;
}

void free_precond(pi_precond* P) {
  if (!P) return;
  for (void* p : P->allocs) cudaFree(p);
  drive_free(P->drive);
  delete P;
}

}  // namespace

cudaError_t precond_apply(const pi_precond* P, const void* r, int r_f32, void* z, int z_f32, double scale,
                          cudaStream_t stream) {
  // the drive state's scratch is written: applications on one plan are serialised by its lock
  if (P->kind == PI_PRECOND_DRIVE) return drive_apply(P->drive, r, r_f32, z, z_f32, stream);
  const PrecondDev& D = P->dev;
  const int blocks = (int)P->host.chain_order.size();
  if (r_f32 != z_f32) return cudaErrorInvalidValue;
  if (P->fp64)
    return r_f32 ? launch_sweep<double, float2, float2>(D, blocks, r, z, scale, stream)
                 : launch_sweep<double, double2, double2>(D, blocks, r, z, scale, stream);
  return r_f32 ? launch_sweep<float, float2, float2>(D, blocks, r, z, scale, stream)
               : launch_sweep<float, double2, double2>(D, blocks, r, z, scale, stream);
}

int precond_coords(const pi_precond* P) { return P->host.coords; }
int precond_kind(const pi_precond* P) { return P->kind; }
double precond_scale(const pi_precond* P) { return P->host.scale; }
const pi_plan* precond_plan(const pi_precond* P) { return P->plan; }

}  // namespace picuda

using namespace picuda;

namespace picuda {
// operator-scale estimate of the plan in the given coordinates (pi_solvers.cu)
int estimate_operator_scale(pi_plan* plan, int coords, double* out);
}  // namespace picuda

extern "C" {

int pi_precond_create(pi_plan* plan, int coords, double regularization, double operator_scale, pi_precond** out) {
  if (!plan || !out) return fail(PI_ERR_INVALID_ARGUMENT, "null argument");
  *out = nullptr;
  if (coords != PI_COORDS_REFERENCE && coords != PI_COORDS_POPULATION)
    return fail(PI_ERR_INVALID_ARGUMENT, "coords must be PI_COORDS_REFERENCE or PI_COORDS_POPULATION");
  if (!(std::isfinite(regularization) && regularization >= 0))
    return fail(PI_ERR_INVALID_ARGUMENT, "regularization must be finite and nonnegative");
  if (operator_scale != 0 && !(std::isfinite(operator_scale) && operator_scale > 0))
    return fail(PI_ERR_INVALID_ARGUMENT, "operator_scale must be finite and positive");
  const auto t0 = std::chrono::steady_clock::now();
  double s = operator_scale;
  if (s == 0) {
    const int rc = estimate_operator_scale(plan, coords, &s);
    if (rc) return rc;
  }
  BusyGuard guard(plan);
  if (!guard.ok) return fail(PI_ERR_BUSY, "a pi_plan cannot be used concurrently");
  pi_precond* P = new pi_precond();
  P->plan = plan;
  P->fp64 = coords == PI_COORDS_REFERENCE ? 1 : 0;
  std::string err;
  int rc = build_level_precond(plan->host, coords, regularization, s, &P->host, &err);
  if (rc) {
    delete P;
    return fail(rc, err);
  }
  const LevelPrecondHost& H = P->host;
  const int* ip = nullptr;
  if ((rc = upload_vec(P, H.chain_order, &ip))) return free_precond(P), rc;
  P->dev.chain_order = ip;
  if ((rc = upload_vec(P, H.chain_lev, &ip))) return free_precond(P), rc;
  P->dev.chain_lev = ip;
  if ((rc = upload_vec(P, H.lev_ent, &ip))) return free_precond(P), rc;
  P->dev.lev_ent = ip;
  if ((rc = upload_vec(P, H.elem, &ip))) return free_precond(P), rc;
  P->dev.elem = ip;
  {
    // the kernel keeps each level in slot order (entry i of a level with K = ceil(cnt / 32)
    // entries per lane at (i mod K) 32 + i / K): store the gain positions as slots of the
    // previous level
    std::vector<int> gslot(H.gsrc.size());
    for (size_t c = 0; c + 1 < H.chain_lev.size(); ++c) {
      for (int lev = H.chain_lev[c]; lev < H.chain_lev[c + 1]; ++lev) {
        const int Kp = lev > H.chain_lev[c] ? (H.lev_ent[lev] - H.lev_ent[lev - 1] + 31) / 32 : 1;
        for (int e = H.lev_ent[lev]; e < H.lev_ent[lev + 1]; ++e) {
          int packed = 0;
          for (int q = 0; q < 3; ++q) {
            int pos = (H.gsrc[e] >> (10 * q)) & 1023;
            pos = pos == kNoGain ? 0 : (pos % Kp) * 32 + pos / Kp;  // none: entry 0, coefficient zero
            packed |= pos << (10 * q);
          }
          gslot[e] = packed;
        }
      }
    }
    if ((rc = upload_vec(P, gslot, &ip))) return free_precond(P), rc;
  }
  P->dev.gsrc = ip;
  rc = P->fp64 ? upload_factors<double>(P) : upload_factors<float>(P);
  if (rc) return free_precond(P), rc;
  const double* dp = nullptr;
  if ((rc = upload_vec(P, H.t0, &dp))) return free_precond(P), rc;
  P->dev.t0 = dp;
  if ((rc = upload_vec(P, H.v0, &dp))) return free_precond(P), rc;
  P->dev.v0 = dp;
  std::vector<double2> w0(H.w0.size());
  for (size_t i = 0; i < w0.size(); ++i) w0[i] = make_double2(H.w0[i].real(), H.w0[i].imag());
  const double2* wp = nullptr;
  if ((rc = upload_vec(P, w0, &wp))) return free_precond(P), rc;
  P->dev.w0 = wp;
  std::vector<float4> w0f(w0.size());  // the same as double-floats (x.hi, x.lo, y.hi, y.lo)
  for (size_t k = 0; k < w0.size(); ++k) {
    const float xh = (float)w0[k].x, yh = (float)w0[k].y;
    w0f[k] = make_float4(xh, (float)(w0[k].x - (double)xh), yh, (float)(w0[k].y - (double)yh));
  }
  const float4* wfp = nullptr;
  if ((rc = upload_vec(P, w0f, &wfp))) return free_precond(P), rc;
  P->dev.w0f = wfp;
  P->dev.chain0 = H.chain0;
  P->dev.chain0_ent = H.chain0_ent;
  P->dev.free_ent = H.free_ent;
  P->dev.mode = H.mode;
  // mode 0: 1 / rho_v
  const std::complex<double> coef = H.mode == 0 ? 1.0 / H.sm_coef : H.sm_coef;
  P->dev.sm_coef = make_double2(coef.real(), coef.imag());
  if (H.free_ent >= 0) P->dev.free_t = H.t0[H.free_ent - H.chain0_ent];
  P->setup_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  *out = P;
  return PI_OK;
}

int pi_precond_create_drive(pi_plan* plan, int coords, double operator_scale, pi_precond** out) {
  if (!plan || !out) return fail(PI_ERR_INVALID_ARGUMENT, "null argument");
  *out = nullptr;
  if (coords != PI_COORDS_REFERENCE && coords != PI_COORDS_POPULATION)
    return fail(PI_ERR_INVALID_ARGUMENT, "coords must be PI_COORDS_REFERENCE or PI_COORDS_POPULATION");
  if (operator_scale != 0 && !(std::isfinite(operator_scale) && operator_scale > 0))
    return fail(PI_ERR_INVALID_ARGUMENT, "operator_scale must be finite and positive");
  double s = operator_scale;
  if (s == 0) {
    const int rc = estimate_operator_scale(plan, coords, &s);
    if (rc) return rc;
  }
  BusyGuard guard(plan);
  if (!guard.ok) return fail(PI_ERR_BUSY, "a pi_plan cannot be used concurrently");
  pi_precond* P = new pi_precond();
  P->plan = plan;
  P->kind = PI_PRECOND_DRIVE;
  P->fp64 = 0;
  P->host.coords = coords;
  P->host.scale = s;
  std::string err;
  const int rc = drive_create(plan, coords, s, &P->drive, &err);
  if (rc) {
    delete P;
    return fail(rc, err);
  }
  P->bytes = drive_bytes(P->drive);
  P->setup_seconds = drive_setup_seconds(P->drive);
  *out = P;
  return PI_OK;
}

int pi_precond_destroy(pi_precond* P) {
  free_precond(P);
  return PI_OK;
}

int pi_precond_info(const pi_precond* P, pi_precond_info_t* out) {
  if (!P || !out) return fail(PI_ERR_INVALID_ARGUMENT, "null argument");
  const LevelPrecondHost& H = P->host;
  out->coords = H.coords;
  out->fp64 = P->fp64;
  out->operator_scale = H.scale;
  out->regularization = H.regularization;
  out->chains = (int)H.chain_order.size();
  out->levels = (int)H.lev_ent.size() - 1;
  out->entries = (long long)H.elem.size();
  out->max_level = H.max_level;
  out->direction = H.direction;
  out->singular = H.mode == 0 ? 1 : 0;
  out->device_bytes = P->bytes;
  out->setup_seconds = P->setup_seconds;
  out->kind = P->kind;
  out->max_asymmetry = 0.0;
  out->max_nonhermitian = 0.0;
  if (P->kind == PI_PRECOND_DRIVE) {
    const DriveHost& D = drive_host(P->drive);
    out->chains = out->levels = out->max_level = out->direction = out->singular = 0;
    out->entries = P->plan->host.dim;
    out->max_asymmetry = D.max_asymmetry;
    out->max_nonhermitian = D.max_nonhermitian;
  }
  return PI_OK;
}

int pi_precond_apply(const pi_precond* P, double* z_dev, const double* r_dev, void* stream) {
  if (!P || !z_dev || !r_dev) return fail(PI_ERR_INVALID_ARGUMENT, "null argument");
  if (z_dev == r_dev) return fail(PI_ERR_INVALID_ARGUMENT, "source and destination must not share storage");
  cudaError_t e = precond_apply(P, r_dev, 0, z_dev, 0, P->host.scale, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_fail(e, "preconditioner apply");
  return PI_OK;
}

}  // extern "C"
