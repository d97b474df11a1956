// Float-float ("double-single") arithmetic on the FP32 pipes: a value is hi + lo with
// |lo| <= ulp(hi)/2, about 48 significant bits.  Algorithms: Dekker's error-free
// transformations (Dekker 1971, "A floating-point technique for extending the available
// precision"; Knuth's TwoSum) as arranged in Bailey/Hida/Li's double-double library, with the
// FMA-based exact product.  GB300 retires FP32 FMAs 64x faster than FP64 ones, so this is how
// the mixed-precision WENO form keeps FP64-class precision in its smoothness indicators and
// nonlinear weights without paying for the FP64 pipe.
#pragma once

#include <cuda_runtime.h>

namespace gbmv {

struct f2 {
  float hi, lo;
  __host__ __device__ constexpr f2() : hi(0.f), lo(0.f) {}
  __host__ __device__ constexpr f2(float h, float l) : hi(h), lo(l) {}
  // from a double constant (split into the nearest float and the rounded remainder)
  __host__ __device__ constexpr explicit f2(double d) : hi((float)d), lo((float)(d - (double)(float)d)) {}
  __host__ __device__ constexpr explicit f2(int i) : hi((float)i), lo(0.f) {}
  __device__ __forceinline__ static f2 from(float x) { return f2(x, 0.f); }
  __device__ __forceinline__ double to_double() const { return (double)hi + (double)lo; }
};

__device__ __forceinline__ f2 quick_two_sum(float a, float b) {  // requires |a| >= |b|
  const float s = a + b;
  return f2(s, b - (s - a));
}

__device__ __forceinline__ f2 two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return f2(s, (a - (s - bb)) + (b - bb));
}

__device__ __forceinline__ f2 two_prod(float a, float b) {
  const float p = a * b;
  return f2(p, fmaf(a, b, -p));
}

__device__ __forceinline__ f2 operator+(f2 x, f2 y) {
  f2 s = two_sum(x.hi, y.hi);
  const float e = s.lo + (x.lo + y.lo);
  return quick_two_sum(s.hi, e);
}
__device__ __forceinline__ f2 operator-(f2 x) { return f2(-x.hi, -x.lo); }
__device__ __forceinline__ f2 operator-(f2 x, f2 y) { return x + (-y); }

__device__ __forceinline__ f2 operator*(f2 x, f2 y) {
  f2 p = two_prod(x.hi, y.hi);
  const float e = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, p.lo));
  return quick_two_sum(p.hi, e);
}

// Division: q1 from a fast approximate reciprocal, the remainder x - y*q1 formed in
// float-float, one correction q2 -- the correction absorbs q1's few-ulp error, so the result
// keeps the float-float precision.
__device__ __forceinline__ f2 operator/(f2 x, f2 y) {
  const float ry = __fdividef(1.f, y.hi);
  const float q1 = x.hi * ry;
  const f2 r = x - y * f2(q1, 0.f);
  const float q2 = r.hi * ry;
  return quick_two_sum(q1, q2);
}

// exact scaling by a power of two
__device__ __forceinline__ f2 f2_scale(f2 x, float p2) { return f2(x.hi * p2, x.lo * p2); }

// exact split of a double into hi + lo (48 of its 53 significant bits survive)
__device__ __forceinline__ f2 f2_from_double(double d) {
  const float h = __double2float_rn(d);
  return f2(h, __double2float_rn(d - (double)h));
}

// Conversions between double and float from the bit patterns, with integer instructions.
// Conversion instructions with a 64-bit operand run at the FP64 rate, 1/64 of the FP32 rate on
// GB300, so in passes that mostly convert (the float-float primitives, the FP32 factors of the
// Newton matrices) they set the time.  Each helper returns exactly what the round-to-nearest
// hardware conversion returns: the integer path covers every normal float result and zeros,
// anything else (subnormal, overflow, inf, NaN) takes the hardware conversion.  In the passes
// bound by the FP64 pipe (f2_split, f2_to_double: RARE) that conversion is a volatile statement:
// the compiler otherwise executes it on every call and selects, and its pipe time is spent after
// all (128^3 x 15: primitives 314 -> 241 us).  The fused Newton is bound by latency: there the
// select is 3 % faster than the branch.
__device__ __forceinline__ float cvt_f32_rare(double d) {
  float f;
  asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(f) : "d"(d));
  return f;
}
__device__ __forceinline__ double cvt_f64_rare(float f) {
  double d;
  asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d) : "f"(f));
  return d;
}

// double -> float, round to nearest even: drop 29 mantissa bits on the pattern (a carry into
// the exponent is the correct rounding), re-bias the exponent (1023 - 127 = 896)
template <bool RARE = false>
__device__ __forceinline__ float f32_of_f64(double d) {
  const unsigned long long p = (unsigned long long)__double_as_longlong(d);
  const unsigned e = (unsigned)(p >> 52) & 0x7FFu;
  if (e - 897u > 1149u - 897u)  // result not surely a normal float: zero, or the conversion
    return !RARE ? __double2float_rn(d)
                 : ((p << 1) == 0 ? __uint_as_float((unsigned)(p >> 32)) : cvt_f32_rare(d));
  const unsigned long long r = p + 0x0FFFFFFFull + ((p >> 29) & 1ull);
  const unsigned hi = (unsigned)(r >> 32);
  const unsigned s = hi & 0x80000000u;
  const unsigned er = (hi >> 20) & 0x7FFu;
  const unsigned m = (unsigned)(r >> 29) & 0x7FFFFFu;
  return __uint_as_float(s | ((er - 896u) << 23) | m);
}

// float -> double, exact
template <bool RARE = false>
__device__ __forceinline__ double f64_of_f32(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xFFu;
  if (e - 1u > 253u)  // zero, or subnormal, inf, NaN
    return !RARE ? (double)f
                 : ((u << 1) == 0 ? __hiloint2double((int)u, 0) : cvt_f64_rare(f));
  const unsigned hi = (u & 0x80000000u) | ((e + 896u) << 20) | ((u & 0x7FFFFFu) >> 3);
  const unsigned lo = u << 29;
  return __hiloint2double((int)hi, (int)lo);
}

// f2_from_double without conversion instructions (bit-identical to it), and for the common
// exponents without the FP64 subtraction either: what rounding to hi leaves of the 53-bit
// significand is a signed integer of 29 bits, whose conversion to float (a 32-bit one) rounds as
// the conversion of the exact difference would.
__device__ __forceinline__ f2 f2_split(double d) {
  const unsigned long long p = (unsigned long long)__double_as_longlong(d);
  const unsigned e = (unsigned)(p >> 52) & 0x7FFu;
  if (e - 949u <= 1149u - 949u) {
    const unsigned long long r = p + 0x0FFFFFFFull + ((p >> 29) & 1ull);
    const unsigned hi = (unsigned)(r >> 32), s = hi & 0x80000000u;
    const unsigned h = s | ((((hi >> 20) & 0x7FFu) - 896u) << 23) | ((unsigned)(r >> 29) & 0x7FFFFFu);
    // p - (r with its low 29 bits cleared), in units of the last place of d
    const int left = (int)((unsigned)p - ((unsigned)r & 0xE0000000u));
    return f2(__uint_as_float(h),
              (float)(s ? -left : left) * __uint_as_float((e - 948u) << 23));
  }
  const float h = f32_of_f64<true>(d);
  return f2(h, f32_of_f64<true>(d - f64_of_f32<true>(h)));
}

// f2::to_double without conversion instructions (bit-identical to it)
__device__ __forceinline__ double f2_to_double(f2 x) {
  return f64_of_f32<true>(x.hi) + f64_of_f32<true>(x.lo);
}

__device__ __forceinline__ bool operator<(f2 a, f2 b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
__device__ __forceinline__ bool operator>(f2 a, f2 b) { return b < a; }
__device__ __forceinline__ bool operator<=(f2 a, f2 b) { return !(b < a); }
__device__ __forceinline__ bool operator==(f2 a, f2 b) { return a.hi == b.hi && a.lo == b.lo; }
__device__ __forceinline__ f2 f2_fabs(f2 a) { return a.hi < 0.f ? -a : a; }

// square root: FP32 estimate, one Newton correction in float-float
__device__ __forceinline__ f2 f2_sqrt(f2 a) {
  if (!(a.hi > 0.f)) return f2(0.f, 0.f);
  const float s = sqrtf(a.hi);
  const f2 ss = two_prod(s, s);
  const float r = ((a.hi - ss.hi) - ss.lo + a.lo) / (2.f * s);
  return quick_two_sum(s, r);
}

}  // namespace gbmv
