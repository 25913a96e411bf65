// Reduction building blocks shared by the Krylov vector kernels (pi_linalg.cu), the engine
// (pi_batch.cu) and the preconditioner sweep (pi_precond.cu).
#pragma once

#include <cuda_runtime.h>

namespace picuda {

// Double-float accumulator: the pair (hi, lo) carries a ~48-bit significand on the FP32
// pipes (GB300 issues FP64 at 1/64 of the FP32 rate).
struct DF {
  float hi, lo;
};

// a += t, the rounding error of the addition carried in a.lo (Knuth's TwoSum).
__device__ __forceinline__ void df_add(DF& a, float t) {
  const float s = a.hi + t;
  const float bb = s - a.hi;
  const float err = (a.hi - (s - bb)) + (t - bb);
  a.hi = s;
  a.lo += err;
}

// acc += a b, the product split exactly with an FMA.
__device__ __forceinline__ void df_add_prod(DF& acc, float a, float b) {
  const float p = a * b;
  const float e = fmaf(a, b, -p);
  const float s = acc.hi + p;
  const float bb = s - acc.hi;
  const float err = (acc.hi - (s - bb)) + (p - bb);
  acc.hi = s;
  acc.lo += err + e;
}

// acc += (ch + cl) v.
__device__ __forceinline__ void df_axpy(DF& acc, float ch, float cl, float v) {
  const float p = ch * v;
  const float e = fmaf(ch, v, -p);
  const float s = acc.hi + p;
  const float bb = s - acc.hi;
  const float err = (acc.hi - (s - bb)) + (p - bb);
  acc.hi = s;
  acc.lo += err + fmaf(cl, v, e);
}

// a + b (TwoSum of the leading parts).
__device__ __forceinline__ DF df_sum(DF a, DF b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float err = (a.hi - (s - bb)) + (b.hi - bb);
  return DF{s, (a.lo + b.lo) + err};
}

// Triple-float accumulator: the sum in hi, the rounding errors of its additions in mid, the errors
// of those in lo (TwoSum twice).  About 70 bits, so a sum of FP32 values or of double-floats is no
// further off than in FP64, and it stays off the FP64 pipe like a double-float.
struct TF {
  float hi, mid, lo;
};
__host__ __device__ __forceinline__ float two_sum(float a, float b, float* err) {
  const float s = a + b;
  const float bb = s - a;
  *err = (a - (s - bb)) + (b - bb);
  return s;
}
__host__ __device__ __forceinline__ void tf_add(TF& a, float t) {
  float e, e2;
  a.hi = two_sum(a.hi, t, &e);
  a.mid = two_sum(a.mid, e, &e2);
  a.lo += e2;
}
__host__ __device__ __forceinline__ double tf_value(const TF& a) {
  return (double)a.hi + ((double)a.mid + (double)a.lo);
}

// Lane sums of NV values (a power of two) by exchanging halves of the values: NV - 1 additions
// and a few more, against 5 NV one value at a time.  Afterwards v[0] of lane l is the total of
// value l / (32 / NV).
template <int NV>
__device__ __forceinline__ void warp_transpose_sum(double (&v)[NV]) {
  const int lane = threadIdx.x & 31;
  int off = 16;
#pragma unroll
  for (int s = NV / 2; s >= 1; s >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < s; ++i) {
      const double send = up ? v[i] : v[i + s];
      const double keep = up ? v[i + s] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  for (; off >= 1; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
}

template <int NV>
__device__ __forceinline__ void warp_transpose_sum(DF (&v)[NV]) {
  const int lane = threadIdx.x & 31;
  int off = 16;
#pragma unroll
  for (int s = NV / 2; s >= 1; s >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < s; ++i) {
      const DF send = up ? v[i] : v[i + s], keep = up ? v[i + s] : v[i];
      v[i] = df_sum(keep, DF{__shfl_xor_sync(0xffffffffu, send.hi, off), __shfl_xor_sync(0xffffffffu, send.lo, off)});
    }
  }
  for (; off >= 1; off >>= 1)
    v[0] = df_sum(v[0], DF{__shfl_xor_sync(0xffffffffu, v[0].hi, off), __shfl_xor_sync(0xffffffffu, v[0].lo, off)});
}

}  // namespace picuda
