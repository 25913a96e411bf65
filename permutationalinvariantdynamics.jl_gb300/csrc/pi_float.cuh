// Sums of FP32 values to more than FP32 precision without the FP64 pipe (GB300 issues FP64 at 1/64 of
// the FP32 rate): pairs and triples of floats.  Plain arithmetic, for device and host alike.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define PI_HD __host__ __device__ __forceinline__
#else
#define PI_HD inline
#endif

namespace picuda {

// Double-float accumulator: the pair (hi, lo) carries a ~48-bit significand on the FP32
// pipes (GB300 issues FP64 at 1/64 of the FP32 rate).
struct DF {
  float hi, lo;
};

// a += t, the rounding error of the addition carried in a.lo (Knuth's TwoSum).
PI_HD void df_add(DF& a, float t) {
  const float s = a.hi + t;
  const float bb = s - a.hi;
  const float err = (a.hi - (s - bb)) + (t - bb);
  a.hi = s;
  a.lo += err;
}

// acc += a b, the product split exactly with an FMA.
PI_HD void df_add_prod(DF& acc, float a, float b) {
  const float p = a * b;
  const float e = fmaf(a, b, -p);
  const float s = acc.hi + p;
  const float bb = s - acc.hi;
  const float err = (acc.hi - (s - bb)) + (p - bb);
  acc.hi = s;
  acc.lo += err + e;
}

// acc += (ch + cl) v.
PI_HD void df_axpy(DF& acc, float ch, float cl, float v) {
  const float p = ch * v;
  const float e = fmaf(ch, v, -p);
  const float s = acc.hi + p;
  const float bb = s - acc.hi;
  const float err = (acc.hi - (s - bb)) + (p - bb);
  acc.hi = s;
  acc.lo += err + fmaf(cl, v, e);
}

// a + b (TwoSum of the leading parts).
PI_HD DF df_sum(DF a, DF b) {
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
PI_HD float two_sum(float a, float b, float* err) {
  const float s = a + b;
  const float bb = s - a;
  *err = (a - (s - bb)) + (b - bb);
  return s;
}
PI_HD void tf_add(TF& a, float t) {
  float e, e2;
  a.hi = two_sum(a.hi, t, &e);
  a.mid = two_sum(a.mid, e, &e2);
  a.lo += e2;
}
PI_HD double tf_value(const TF& a) {
  return (double)a.hi + ((double)a.mid + (double)a.lo);
}

// a + b of double-floats, and of triple-floats.
PI_HD TF tf_pair(DF a, DF b) {
  float e, e2, e3;
  const float s = two_sum(a.hi, b.hi, &e);
  const float m = two_sum(two_sum(a.lo, b.lo, &e2), e, &e3);
  return TF{s, m, e2 + e3};
}
PI_HD TF tf_sum(const TF& a, const TF& b) {
  float e, e2, e3;
  const float s = two_sum(a.hi, b.hi, &e);
  const float m = two_sum(two_sum(a.mid, b.mid, &e2), e, &e3);
  return TF{s, m, (a.lo + b.lo) + (e2 + e3)};
}

}  // namespace picuda
