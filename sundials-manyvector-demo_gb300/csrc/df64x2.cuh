// Two independent float-float numbers side by side: lane x and lane y of float2 registers,
// operated on with the paired FP32 instructions of sm_100-class GPUs (__fadd2_rn, __fmul2_rn,
// __ffma2_rn: one instruction performs the same IEEE round-to-nearest operation on both
// lanes).  Every operator below is the df64.cuh algorithm of the same name applied to each
// lane, so lane x of a result equals, bit for bit, what the scalar f2 operation returns for
// the lane-x operands (and likewise for y), in half the FP32 instructions.
//
// Used where the WENO face flux evaluates the same formula twice on different data: the two
// Lax-Friedrichs sides of every reconstruction (the minus side's stencil reversed, which turns
// its formula into the plus side's).
#pragma once

#include <cuda_runtime.h>

#include "df64.cuh"

namespace gbmv {

__device__ __forceinline__ float2 v2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

struct f2v {
  float2 hi, lo;
  __device__ __forceinline__ f2v() : hi(make_float2(0.f, 0.f)), lo(make_float2(0.f, 0.f)) {}
  __device__ __forceinline__ f2v(float2 h, float2 l) : hi(h), lo(l) {}
  // lane x = a, lane y = b
  __device__ __forceinline__ f2v(f2 a, f2 b) : hi(make_float2(a.hi, b.hi)), lo(make_float2(a.lo, b.lo)) {}
  // the same value in both lanes
  __device__ __forceinline__ explicit f2v(f2 a) : hi(v2(a.hi)), lo(v2(a.lo)) {}
  __device__ __forceinline__ f2 x() const { return f2(hi.x, lo.x); }
  __device__ __forceinline__ f2 y() const { return f2(hi.y, lo.y); }
};

__device__ __forceinline__ f2v quick_two_sum2(float2 a, float2 b) {  // |a| >= |b| per lane
  const float2 s = add2(a, b);
  return f2v(s, sub2(b, sub2(s, a)));
}

__device__ __forceinline__ f2v two_sum2(float2 a, float2 b) {
  const float2 s = add2(a, b);
  const float2 bb = sub2(s, a);
  return f2v(s, add2(sub2(a, sub2(s, bb)), sub2(b, bb)));
}

__device__ __forceinline__ f2v two_prod2(float2 a, float2 b) {
  const float2 p = mul2(a, b);
  return f2v(p, fma2(a, b, neg2(p)));
}

__device__ __forceinline__ f2v operator+(f2v x, f2v y) {
  const f2v s = two_sum2(x.hi, y.hi);
  const float2 e = add2(s.lo, add2(x.lo, y.lo));
  return quick_two_sum2(s.hi, e);
}
__device__ __forceinline__ f2v operator-(f2v x) { return f2v(neg2(x.hi), neg2(x.lo)); }
__device__ __forceinline__ f2v operator-(f2v x, f2v y) { return x + (-y); }

__device__ __forceinline__ f2v operator*(f2v x, f2v y) {
  const f2v p = two_prod2(x.hi, y.hi);
  const float2 e = fma2(x.hi, y.lo, fma2(x.lo, y.hi, p.lo));
  return quick_two_sum2(p.hi, e);
}

// Pieces without the final renormalisation (|lo| a few ulps of hi instead of half of one), for
// values that are only multiplied or summed with others of their sign afterwards: a product in 4
// operations instead of 7, a product added to a sum in 12 instead of 18.
__device__ __forceinline__ f2v f2v_prod(f2v x, f2v y) {
  const f2v p = two_prod2(x.hi, y.hi);
  return f2v(p.hi, fma2(x.hi, y.lo, fma2(x.lo, y.hi, p.lo)));
}
__device__ __forceinline__ f2v f2v_add_prod(f2v s, f2v x, f2v y) {  // s + x y
  const f2v p = two_prod2(x.hi, y.hi);
  const f2v t = two_sum2(s.hi, p.hi);
  const float2 e = add2(add2(s.lo, t.lo), p.lo);
  return f2v(t.hi, fma2(x.hi, y.lo, fma2(x.lo, y.hi, e)));
}
__device__ __forceinline__ f2v f2v_sum(f2v x, f2v y) {  // x + y
  const f2v s = two_sum2(x.hi, y.hi);
  return f2v(s.hi, add2(s.lo, add2(x.lo, y.lo)));
}
__device__ __forceinline__ f2v f2v_norm(f2v x) { return quick_two_sum2(x.hi, x.lo); }
// x y + z
__device__ __forceinline__ f2v f2v_fma(f2v x, f2v y, f2v z) {
  return f2v_norm(f2v_add_prod(z, x, y));
}
// x / y from the approximate reciprocal, one residual (its leading part exact in an FMA) and one
// correction: 10 operations where one with the remainder in float-float takes 25
__device__ __forceinline__ f2v f2v_quot(f2v x, f2v y) {
  const float2 r = make_float2(__fdividef(1.f, y.hi.x), __fdividef(1.f, y.hi.y));
  const float2 q = mul2(x.hi, r), n = neg2(q);
  const float2 t = fma2(y.lo, n, add2(fma2(y.hi, n, x.hi), x.lo));
  return quick_two_sum2(q, mul2(t, r));
}

// exact scaling by a power of two
__device__ __forceinline__ f2v f2v_scale(f2v x, float p2) {
  return f2v(mul2(x.hi, v2(p2)), mul2(x.lo, v2(p2)));
}

}  // namespace gbmv
