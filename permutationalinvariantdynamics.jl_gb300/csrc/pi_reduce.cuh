// Reduction building blocks shared by the Krylov vector kernels (pi_linalg.cu), the engine
// (pi_batch.cu) and the preconditioner sweep (pi_precond.cu).
#pragma once

#include <cuda_runtime.h>

#include "pi_float.cuh"

namespace picuda {

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

// The same for double-floats, exactly enough that the lane sums add nothing to the error of the
// accumulators (pi_float.cuh): v[0] of lane l in triple-float.
template <int NV>
__device__ __forceinline__ TF warp_transpose_total(const DF (&v)[NV]) {
  static_assert(NV >= 2, "the first exchange halves the values");
  const int lane = threadIdx.x & 31;
  const bool up = lane & 16;
  TF t[NV / 2];
#pragma unroll
  for (int i = 0; i < NV / 2; ++i) {
    const DF send = up ? v[i] : v[i + NV / 2], keep = up ? v[i + NV / 2] : v[i];
    t[i] = tf_pair(keep, DF{__shfl_xor_sync(0xffffffffu, send.hi, 16), __shfl_xor_sync(0xffffffffu, send.lo, 16)});
  }
  auto other = [](const TF& a, int off) {
    return TF{__shfl_xor_sync(0xffffffffu, a.hi, off), __shfl_xor_sync(0xffffffffu, a.mid, off),
              __shfl_xor_sync(0xffffffffu, a.lo, off)};
  };
#pragma unroll
  for (int step = 1; step < 5; ++step) {
    const int off = 16 >> step, left = NV >> (step + 1);  // values left after this step (0: one, summed on)
    const bool high = lane & off;
    if (left == 0) {
      t[0] = tf_sum(t[0], other(t[0], off));
      continue;
    }
#pragma unroll
    for (int i = 0; i < left; ++i) {
      const TF send = high ? t[i] : t[i + left], keep = high ? t[i + left] : t[i];
      t[i] = tf_sum(keep, other(send, off));
    }
  }
  return t[0];
}

}  // namespace picuda
