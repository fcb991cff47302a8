// tlr_ff.cuh -- float-float arithmetic (Dekker / Knuth error-free
// transformations on FP32): a value is hi + lo, about 48 bits.
#pragma once

#include <cuda_runtime.h>

namespace tlr {

// (hi, lo) += a * x with a = ah + al, x = xh + xl
__device__ __forceinline__ void ff_mac(float &hi, float &lo, float ah, float al, float xh,
                                       float xl) {
  const float p = ah * xh;
  const float e = fmaf(ah, xh, -p) + fmaf(ah, xl, al * xh);
  const float s = hi + p;
  const float bb = s - hi;
  lo += ((hi - (s - bb)) + (p - bb)) + e;
  hi = s;
}

__device__ __forceinline__ void ff_add(float &hi, float &lo, float h2, float l2) {
  const float s = hi + h2;
  const float bb = s - hi;
  lo = lo + l2 + ((hi - (s - bb)) + (h2 - bb));
  hi = s;
}

// (re_hi, re_lo, im_hi, im_lo) of a complex128 value
__device__ __forceinline__ float4 ff_split(double2 v) {
  const float rh = __double2float_rn(v.x), ih = __double2float_rn(v.y);
  return make_float4(rh, __double2float_rn(v.x - (double)rh), ih,
                     __double2float_rn(v.y - (double)ih));
}

// a complex accumulator: (h, l) pairs of the real and imaginary part
struct FFC {
  float rh, rl, ih, il;
};

// acc += a x (complex)
__device__ __forceinline__ void ffc_mac(FFC &s, const float4 &a, const float4 &x) {
  ff_mac(s.rh, s.rl, a.x, a.y, x.x, x.y);
  ff_mac(s.rh, s.rl, -a.z, -a.w, x.z, x.w);
  ff_mac(s.ih, s.il, a.x, a.y, x.z, x.w);
  ff_mac(s.ih, s.il, a.z, a.w, x.x, x.y);
}

__device__ __forceinline__ double2 ffc_value(const FFC &s) {
  return make_double2((double)s.rh + (double)s.rl, (double)s.ih + (double)s.il);
}

}  // namespace tlr
