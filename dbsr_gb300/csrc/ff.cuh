// ff.cuh -- float-float arithmetic for the gather-sums of the split form.
//
// A value v is carried as two FP32 numbers (hi, lo) with hi = fl32(v) and
// lo = fl32(v - hi): 48 significant bits.  A gather-sum S = sum_e c_e K_e
// (25-60 terms here) is accumulated as
//   p  = hi(c) hi(K)                     rounded product
//   pe = fma(hi(c), hi(K), -p)           its exact rounding error (TwoProd)
//   x  = hi(c) lo(K) + lo(c) hi(K) + pe  the small terms, in FP32
//   (s_hi, e) = TwoSum(s_hi, p)          exact (Knuth, six additions)
//   s_lo += e + x
// so every product is exact to about 2^-48 of itself and the sum to about
// (terms) x 2^-48 of sum |c_e K_e| -- far inside the 1e-10 per-block bound of
// the split form, at FP32 instruction rates (GB300's FP64 pipe runs about
// 2 operations per clock per SM).  The compiler may contract a*b+c into
// FMA; the TwoSum contains no product, so contraction leaves it exact.
#pragma once
#include <cuda_runtime.h>

namespace ffa {

// Conversions between double and float-float in integer arithmetic: the 64-bit
// conversion instructions run on the FP64 pipe at about two a clock and SM, and
// a split takes three of its instructions, a sum of two floats three more.
// hi: the bits rounded to 24 (ties away from zero); lo: what is left, a signed
// integer of 29 bits, converted and scaled by v's power of two in two exact
// steps.  Values past the ends of the normal floats take the conversion.
__device__ __forceinline__ float2 split(double v) {
  const unsigned hw = (unsigned)__double2hiint(v), lw = (unsigned)__double2loint(v);
  const unsigned e = hw >> 20 & 0x7ffu, sign = hw & 0x80000000u;
  if (e - 898u > 251u) {
    // below half the smallest float: zero; below 2^-125 the rest of the rounded
    // value is less than half the smallest float
    if (e < 873u) return make_float2(__uint_as_float(sign), 0.0f);
    const float h = __double2float_rn(v);
    if (e < 898u) return make_float2(h, 0.0f);
    return make_float2(h, __double2float_rn(v - (double)h));
  }
  const unsigned lr = lw + 0x10000000u, hr = hw + (lr < lw ? 1u : 0u);
  // the exponent field's low nine bits above the 23 of the mantissa, 1023 - 127
  // taken off modulo 512
  const unsigned h = ((hr << 3 | lr >> 29) - 0xC0000000u) | sign;
  const int rem = (int)(lr & 0x1fffffffu) - 0x10000000;
  const float p2 = __uint_as_float((e - 896u) << 23 | sign);
  return make_float2(__uint_as_float(h), (float)rem * 0x1p-52f * p2);
}

__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f), a = b & 0x7fffffffu;
  if (a - 0x00800000u >= 0x7f000000u && a != 0) return (double)f;
  const unsigned h = a ? (a >> 3) + 0x38000000u : 0u;
  return __hiloint2double((int)(h | (b & 0x80000000u)), (int)(b << 29));
}

__device__ __forceinline__ void mac(float2 c, float2 k, float &sh, float &sl) {
  const float p = c.x * k.x;
  const float pe = fmaf(c.x, k.x, -p);
  const float x = fmaf(c.x, k.y, fmaf(c.y, k.x, pe));
  const float s = sh + p;
  const float bp = s - sh;
  const float e = (sh - (s - bp)) + (p - bp);
  sh = s;
  sl = sl + (e + x);
}

// (sh, sl) += v for a float-float v (TwoSum of the high parts)
__device__ __forceinline__ void add(float2 v, float &sh, float &sl) {
  const float s = sh + v.x;
  const float bp = s - sh;
  const float e = (sh - (s - bp)) + (v.x - bp);
  sh = s;
  sl = sl + (e + v.y);
}

__device__ __forceinline__ double value(float sh, float sl) { return widen(sh) + widen(sl); }

// (hi, lo) renormalised so that lo is below half an ulp of hi (Fast2Sum)
__device__ __forceinline__ float2 norm(float sh, float sl) {
  const float s = sh + sl;
  return make_float2(s, sl - (s - sh));
}

}  // namespace ffa

// a sum and its terms in either arithmetic: float-float (FF) or FP64
template <bool FF>
struct Val;
template <>
struct Val<true> {
  using T = float2;
  float h = 0.0f, l = 0.0f;
  __device__ void mac(float2 a, float2 b) { ffa::mac(a, b, h, l); }
  __device__ void add_value(float2 o) { ffa::add(o, h, l); }
  // the low sum back below half an ulp of the high one: its own rounding errors
  // grow with its size, which is a random walk over the terms added
  __device__ void renorm() {
    const float2 v = ffa::norm(h, l);
    h = v.x;
    l = v.y;
  }
  __device__ float2 get() const { return ffa::norm(h, l); }
  __device__ double value() const { return ffa::value(h, l); }
  __device__ static float2 zero() { return make_float2(0.0f, 0.0f); }
  __device__ static float2 of(double v) { return ffa::split(v); }
  __device__ static double dbl(float2 v) { return ffa::value(v.x, v.y); }
  __device__ static float2 mul(float2 a, float2 b) {
    const float p = a.x * b.x;
    const float e = fmaf(a.x, b.x, -p);
    return ffa::norm(p, fmaf(a.x, b.y, fmaf(a.y, b.x, e)));
  }
};
template <>
struct Val<false> {
  using T = double;
  double v = 0.0;
  __device__ void mac(double a, double b) { v = fma(a, b, v); }
  __device__ void add_value(double o) { v += o; }
  __device__ void renorm() {}
  __device__ double get() const { return v; }
  __device__ double value() const { return v; }
  __device__ static double zero() { return 0.0; }
  __device__ static double of(double x) { return x; }
  __device__ static double dbl(double x) { return x; }
  __device__ static double mul(double a, double b) { return a * b; }
};
