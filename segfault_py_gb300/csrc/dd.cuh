// dd.cuh -- double-float ("dd") arithmetic on the FP32 pipe.
//
// A value is the unevaluated sum hi + lo of two floats with |lo| <= ulp(hi)/2,
// about 48 significant bits.  GB300's FP64 pipe runs at 1/64 of the FP32 rate
// and one warp's FP64 instruction occupies its sub-partition's FP64 unit for
// 64 cycles, so a quartet evaluated with dd operations (7 to 15 FP32
// instructions each) is several times faster than the same quartet in FP64,
// with a relative rounding error near 2^-44 instead of 2^-53.
//
// The building blocks are the error-free transformations of Knuth (TwoSum),
// Dekker (FastTwoSum) and the FMA form of TwoProduct; the "sloppy" addition
// and the multiplication follow the double-double algorithms of Hida, Li and
// Bailey (QD library paper, 2001), written here for float pairs.  The leading
// product of each is __fmul_rn: a plain one may be contracted into a following
// addition, whose rounding error the transformation then no longer captures.
#pragma once
#include <cuda_runtime.h>

namespace sf {

struct dd {
  float hi, lo;
  dd() = default;
  __host__ __device__ constexpr dd(float h, float l) : hi(h), lo(l) {}
  __host__ __device__ constexpr dd(float h) : hi(h), lo(0.0f) {}
  __host__ __device__ constexpr dd(int i) : hi((float)i), lo(0.0f) {}
  // split of a double (constant-folded for compile-time constants)
  __host__ __device__ constexpr explicit dd(double d) : hi((float)d), lo((float)(d - (double)(float)d)) {}
};

__device__ __forceinline__ dd dd_fast_two_sum(float a, float b) {   // |a| >= |b|
  const float s = a + b;
  return dd(s, b - (s - a));
}

__device__ __forceinline__ dd dd_two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return dd(s, (a - (s - bb)) + (b - bb));
}

__device__ __forceinline__ dd operator+(dd a, dd b) {
  dd s = dd_two_sum(a.hi, b.hi);
  return dd_fast_two_sum(s.hi, s.lo + (a.lo + b.lo));
}
__device__ __forceinline__ dd operator-(dd a) { return dd(-a.hi, -a.lo); }
__device__ __forceinline__ dd operator-(dd a, dd b) { return a + (-b); }

__device__ __forceinline__ dd operator*(dd a, dd b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return dd_fast_two_sum(p, e);
}
__device__ __forceinline__ dd operator*(dd a, float b) {
  const float p = __fmul_rn(a.hi, b);
  float e = fmaf(a.hi, b, -p);
  e = fmaf(a.lo, b, e);
  return dd_fast_two_sum(p, e);
}
__device__ __forceinline__ dd operator*(float b, dd a) { return a * b; }
__device__ __forceinline__ dd operator*(dd a, int b) { return a * (float)b; }
__device__ __forceinline__ dd operator*(int b, dd a) { return a * (float)b; }

// a*b + c with one renormalisation
__device__ __forceinline__ dd dd_fma(dd a, dd b, dd c) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  dd s = dd_two_sum(p, c.hi);
  return dd_fast_two_sum(s.hi, s.lo + (e + c.lo));
}

__device__ __forceinline__ dd dd_fma(float a, dd b, dd c) {
  const float p = __fmul_rn(a, b.hi);
  float e = fmaf(a, b.hi, -p);
  e = fmaf(a, b.lo, e);
  dd s = dd_two_sum(p, c.hi);
  return dd_fast_two_sum(s.hi, s.lo + (e + c.lo));
}

// a*b + c for |c| >= |a b|
__device__ __forceinline__ dd dd_fma_big(dd a, dd b, dd c) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  dd s = dd_fast_two_sum(c.hi, p);
  return dd_fast_two_sum(s.hi, s.lo + (e + c.lo));
}

__device__ __forceinline__ dd &operator+=(dd &a, dd b) { return a = a + b; }
__device__ __forceinline__ dd &operator-=(dd &a, dd b) { return a = a - b; }
__device__ __forceinline__ dd &operator*=(dd &a, dd b) { return a = a * b; }
__device__ __forceinline__ dd &operator*=(dd &a, float b) { return a = a * b; }

__device__ __forceinline__ bool operator>=(dd a, float b) { return a.hi > b || (a.hi == b && a.lo >= 0.0f); }

// a*b without the renormalisation: |lo| up to two units of hi's last place,
// for a factor of dd_acc
__device__ __forceinline__ dd dd_mul_raw(dd a, dd b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return dd(p, e);
}

// s += a*b for a sum that stays unnormalised (lo gathers the rounding of hi
// and of the products): 12 instructions, a multiplication and an addition with
// their renormalisations take 18.  dd_norm before anything but another dd_acc.
__device__ __forceinline__ void dd_acc(dd &s, dd a, dd b) {
  const dd m = dd_mul_raw(a, b);
  const dd t = dd_two_sum(s.hi, m.hi);
  s = dd(t.hi, s.lo + (t.lo + m.lo));
}
__device__ __forceinline__ dd dd_norm(dd a) { return dd_two_sum(a.hi, a.lo); }

// 1 - a for 0 <= a <= 1
__device__ __forceinline__ dd dd_one_minus(dd a) {
  const dd s = dd_fast_two_sum(1.0f, -a.hi);
  return dd_fast_two_sum(s.hi, s.lo - a.lo);
}

// k*a for a small integer k (2 a is exact)
__device__ __forceinline__ dd dd_times(int k, dd a) {
  return k == 1 ? a : k == 2 ? dd(2.0f * a.hi, 2.0f * a.lo) : a * (float)k;
}

// 1/a: FP32 reciprocal seed y, residual 1 - a y = r - e (r exact, e its FP32
// rounding terms, about 2^-24): y + y (r - e) + y (r - e)^2, the product y r exact;
// relative error 2e-15 rms, 1.4e-14 at most (4e6 values, seeds within 2 ulp)
__device__ __forceinline__ dd dd_recip(dd a) {
  const float y = 1.0f / a.hi;
  const float p = __fmul_rn(a.hi, y);
  const float e = fmaf(a.lo, y, fmaf(a.hi, y, -p));
  const float r = 1.0f - p, t = r - e;
  const float c = __fmul_rn(y, r);
  const float d = fmaf(y, r, -c) + y * fmaf(t, t, -e);
  const dd s = dd_fast_two_sum(y, c);
  return dd_fast_two_sum(s.hi, s.lo + d);
}

// 1/sqrt(a): FP32 seed y, residual 1 - a y^2 = r - e (r exact), then
// y + y (r - e) / 2 + 3/8 y (r - e)^2, the product y r / 2 exact: relative error 1.4e-15
// rms, 1.6e-14 at most (4e6 values, seeds within 2 ulp).  The 1/(p+q) in the Rys argument
// x amplifies it by x, but e in double-float (6e-16 rms) changed the errors of J, K and
// forces (mean of 13 molecules) by up to 8 % either way and cost 1.5 %.
__device__ __forceinline__ dd dd_rsqrt(dd a) {
  const float y = rsqrtf(a.hi);
  const float q = __fmul_rn(y, y), ql = fmaf(y, y, -q);
  const float p = __fmul_rn(a.hi, q);
  float e = fmaf(a.hi, q, -p);
  e = fmaf(a.hi, ql, e);
  e = fmaf(a.lo, q, e);
  const float r = 1.0f - p, h = 0.5f * r, t = r - e;
  const float c = __fmul_rn(y, h);
  const float d = fmaf(y, h, -c) + y * (0.375f * t * t - 0.5f * e);
  const dd s = dd_fast_two_sum(y, c);
  return dd_fast_two_sum(s.hi, s.lo + d);
}

__device__ __forceinline__ dd dd_shfl_xor(unsigned mask, dd v, int lane_mask) {
  return dd(__shfl_xor_sync(mask, v.hi, lane_mask), __shfl_xor_sync(mask, v.lo, lane_mask));
}

__device__ __forceinline__ dd dd_ldg(const dd *p) {
  const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
  return dd(v.x, v.y);
}

}  // namespace sf
