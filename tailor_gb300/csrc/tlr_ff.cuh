// tlr_ff.cuh -- float-float arithmetic (Dekker / Knuth error-free
// transformations on FP32): a value is hi + lo, about 48 bits.
#pragma once

#include <cuda_runtime.h>

namespace tlr {

// (hi, lo) += a * x with a = ah + al, x = xh + xl: the leading product is
// exact in p + e, its sum exact in s and the two-sum's rest; twelve
// instructions
__device__ __forceinline__ void ff_mac(float &hi, float &lo, float ah, float al, float xh,
                                       float xl) {
  const float p = __fmul_rn(ah, xh);
  const float e = fmaf(ah, xh, -p);
  lo = fmaf(ah, xl, lo);
  lo = fmaf(al, xh, lo);
  const float s = __fadd_rn(hi, p);
  const float bb = __fadd_rn(s, -hi);
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

// (h, l) with h + l renormalised so that h carries the leading bits
__device__ __forceinline__ void ff_norm(float &h, float &l) {
  const float s = h + l;
  l = l - (s - h);
  h = s;
}

// a - b of two complex float-float values
__device__ __forceinline__ float4 ffc_sub(float4 a, const FFC &b) {
  ff_add(a.x, a.y, -b.rh, -b.rl);
  ff_add(a.z, a.w, -b.ih, -b.il);
  ff_norm(a.x, a.y);
  ff_norm(a.z, a.w);
  return a;
}

// a * f, f = fh + fl real
__device__ __forceinline__ float4 ffc_scale(float4 a, float fh, float fl) {
  float4 r;
  r.x = a.x * fh;
  r.y = fmaf(a.x, fh, -r.x) + fmaf(a.x, fl, a.y * fh);
  r.z = a.z * fh;
  r.w = fmaf(a.z, fh, -r.z) + fmaf(a.z, fl, a.w * fh);
  ff_norm(r.x, r.y);
  ff_norm(r.z, r.w);
  return r;
}

__device__ __forceinline__ double2 ff_value(const float4 &a) {
  return make_double2((double)a.x + (double)a.y, (double)a.z + (double)a.w);
}

__device__ __forceinline__ double2 ffc_value(const FFC &s) {
  return make_double2((double)s.rh + (double)s.rl, (double)s.ih + (double)s.il);
}

}  // namespace tlr
