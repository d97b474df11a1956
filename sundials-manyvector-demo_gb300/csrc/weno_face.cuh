// WENO5 face flux in float-float arithmetic (~48-bit significand) on the FP32 pipes -- the mixed
// forms of the reference's face_flux (src/utilities.cpp:270-479).  GB300 retires FP32 FMAs 64x
// faster than FP64 ones, and the reference's eigenvector basis (built with c^2 where c is expected,
// src/utilities.cpp:309) is ill-conditioned when c is small in code units, so plain FP32
// characteristic arithmetic loses too many digits; float-float keeps FP64-class accuracy.  Values
// beyond 1e18 in magnitude (where a float square would overflow) fall back to native FP64.
//
// The arrangement is weno64.cuh's (reconstruction as central value plus correction from neighbour
// differences, both Lax-Friedrichs sides as products with (u +- alpha)/2, shared eigenvector
// terms), because here too the operations set the time: a float-float addition is 11 FP32
// instructions, a product 7.  Both sides of a face are the two lanes of the paired FP32
// instructions (df64x2.cuh), the minus side's stencil reversed, which turns its formula into the
// plus side's.
#pragma once

#include "common.cuh"
#include "df64.cuh"
#include "df64x2.cuh"
#include "weno64.cuh"

namespace gbmv {

__device__ __forceinline__ f2 f2_sqrt0(f2 x) { return x <= f2(0.0) ? f2(0.0) : f2_sqrt(x); }

// a + b as floats: the leading part of the float-float difference a - b
__device__ __forceinline__ float2 f2v_diff_hi(f2v a, f2v b) {
  const f2v s = two_sum2(a.hi, neg2(b.hi));
  return add2(s.hi, add2(s.lo, sub2(a.lo, b.lo)));
}
__device__ __forceinline__ f2v f2v_times(float c, f2v y) {  // c y, not renormalised
  const f2v p = two_prod2(v2(c), y.hi);
  return f2v(p.hi, fma2(v2(c), y.lo, p.lo));
}
__device__ __forceinline__ f2v f2v_add_scaled(f2v s, float c, f2v y) {  // s + c y
  const f2v p = two_prod2(v2(c), y.hi);
  const f2v t = two_sum2(s.hi, p.hi);
  return f2v(t.hi, fma2(v2(c), y.lo, add2(add2(s.lo, t.lo), p.lo)));
}

// Power of two that brings the product of the two largest of three positive values to ~1
__device__ __forceinline__ float weno_scale(float a, float b, float c) {
  const int ea = __float_as_int(a) >> 23, eb = __float_as_int(b) >> 23,
            ec = __float_as_int(c) >> 23;
  const int two = ea + eb + ec - min(ea, min(eb, ec)) - 254;
  return __int_as_float((127 - two / 2) << 23);
}

// The float-float reconstructions work on kF2Scale times the fluxes (the split factors and the
// pressure carry it, so it costs nothing there): the weights' numerator holds eps^4 times a flux
// difference, whose low part would leave the float range for small fluxes.  Scaled so that eps is
// near 1 (0.79), the numerator leaves it where the fluxes' own float pairs do.  (Scale 64: errors
// of 1e-7 at fluxes of 1e-30, 1e-3 at 1e-34; 1024: 2e-14 and 7e-11, as ratios of the a_k had.)
constexpr float kF2Scale = 1024.f;

// Both reconstructions of a face (lane x the plus side, lane y the minus side with its stencil
// reversed), values scaled by s in and out, s2 = s^2: weno_diff64's formula.  The weights' products hold a^4 and
// the numerator a candidate's correction beside it.  With a_k <= A, every |D23| and |D12| is below
// 1.29 sqrt(A) and |D34|, |D01| below 2.77 sqrt(A), so |cA| + |cB| + |cC| < 9.8 sqrt(A) and the
// numerator stays below 9.8 A^4.5: 2^125 for A = 2^27 (the denominator below 10 A^4 = 2^112).
// Beyond, the a_k are scaled by a common power of two, which the weights do not see.  One
// out-of-line copy serves every reconstruction of a face (the kernel stays inside the instruction
// cache).
constexpr float kF2Big = 134217728.f;  // 2^27
static __device__ __noinline__ f2v weno_plus_f2v(f2v f0, f2v f1, f2v f2_, f2v f3, f2v f4,
                                                 float s2) {
  const f2v D01 = f0 - f1, D12 = f1 - f2_, D23 = f2_ - f3, D34 = f3 - f4;
  const f2v D23x2 = f2v_scale(D23, 2.f);
  f2v aA, aB, aC;
  {
    // (the t's and k's are not renormalised: they only go into products, and what those drop
    // stays below 2^-48 of a_k)
    const f2v eps = f2v_scale(f2v(f2(kWenoEps)), s2);
    const f2v s23 = f2v_add_prod(eps, f2v_times(39.f / 64.f, D23), D23);
    const f2v s12 = f2v_add_prod(eps, f2v_times(39.f / 64.f, D12), D12);
    const f2v tA = f2v_add_scaled(D34, -11.f / 8.f, D23), tB = f2v_add_scaled(D12, -5.f / 8.f, D23),
              tC = f2v_add_scaled(D01, -11.f / 8.f, D12);
    aA = f2v_norm(f2v_add_prod(s23, tA, tA));
    aB = f2v_norm(f2v_add_prod(s23, tB, tB));
    aC = f2v_norm(f2v_add_prod(s12, tC, tC));
  }
  const float top = fmaxf(fmaxf(fmaxf(aA.hi.x, aB.hi.x), aC.hi.x),
                          fmaxf(fmaxf(aA.hi.y, aB.hi.y), aC.hi.y));
  if (top > kF2Big) {
    const float2 s = make_float2(weno_scale(aA.hi.x, aB.hi.x, aC.hi.x),
                                 weno_scale(aA.hi.y, aB.hi.y, aC.hi.y));
    aA = f2v(mul2(aA.hi, s), mul2(aA.lo, s));
    aB = f2v(mul2(aB.hi, s), mul2(aB.lo, s));
    aC = f2v(mul2(aC.hi, s), mul2(aC.lo, s));
  }
  const f2v PA = f2v_prod(aB, aC), PB = f2v_prod(aA, aC), PC = f2v_prod(aA, aB);
  const f2v sA = f2v_prod(PA, PA), sB = f2v_prod(PB, PB), sC = f2v_prod(PC, PC);
  const f2v den = f2v_norm(f2v_add_scaled(f2v_add_scaled(sC, 3.f, sA), 6.f, sB));
  // 3 sA (qA - f2) + 6 sB (qB - f2) + sC (qC - f2)
  const f2v cA = f2v_sum(f2v_scale(D34, 0.5f), -D23x2), cB = -f2v_sum(D12, D23x2);
  const f2v cC = f2v_add_prod(f2v_prod(f2v(f2(1.0 / 3.0)), D01), f2v(f2(-5.0 / 6.0)), D12);
  const f2v num = f2v_norm(f2v_add_prod(f2v_add_prod(f2v_prod(sA, cA), sB, cB), sC, cC));
  return f2_ + f2v_quot(num, den);
}

// Reconstruction in correction form with FP32 weights (GBMV_MIXED_FAST, species fields): with the
// central point f2_ in float-float, r = f2_ + sum_k w_k (q_k - f2_).  The corrections q_k - f2_ and
// the smoothness indicators are built from the neighbour differences D01..D34 (exact float-float
// subtractions, then rounded to float), and the weights and the weighted correction are FP32: a
// relative weight error e changes r by e |q_k - f2_| -- an O(dx) difference in smooth flow, the
// jump across a discontinuity -- never by e |r|, because the base value is not weighted (the three
// weights need not sum to exactly one).  Used for the componentwise species reconstructions only:
// the characteristic values of the fluid part are back-projected through an eigenbasis with
// condition ~1/c^2, which would amplify the weight rounding (measured: 2e-5 on the chem-hydro
// state).
__device__ __forceinline__ f2v weno_plus_f2dv(f2v f0, f2v f1, f2v f2_, f2v f3, f2v f4) {
  const float2 D01 = f2v_diff_hi(f0, f1), D12 = f2v_diff_hi(f1, f2_), D23 = f2v_diff_hi(f2_, f3),
               D34 = f2v_diff_hi(f3, f4);
  const float2 dA = sub2(D23, D34), dB = sub2(D12, D23), dC = sub2(D01, D12);
  const float2 eA = fma2(v2(2.f), D23, dA), eB = add2(D12, D23), eC = fma2(v2(-2.f), D12, dC);
  const float2 b13 = v2(13.f / 12.f), q = v2(0.25f), sixth = v2(1.f / 6.f);
  const float2 aA = add2(v2(1e-6f), fma2(b13, mul2(dA, dA), mul2(q, mul2(eA, eA))));
  const float2 aB = add2(v2(1e-6f), fma2(b13, mul2(dB, dB), mul2(q, mul2(eB, eB))));
  const float2 aC = add2(v2(1e-6f), fma2(b13, mul2(dC, dC), mul2(q, mul2(eC, eC))));
  // candidate minus central point (plus side: linear weights 0.3, 0.6, 0.1)
  const float2 cA = mul2(fma2(v2(-4.f), D23, D34), sixth);
  const float2 cB = mul2(fma2(v2(2.f), D23, D12), v2(-1.f / 6.f));
  const float2 cC = mul2(fma2(v2(-5.f), D12, mul2(v2(2.f), D01)), sixth);
  const float2 m = make_float2(fminf(fminf(aA.x, aB.x), aC.x), fminf(fminf(aA.y, aB.y), aC.y));
  // ratios in (0, 1] and a sum of weights above 0.1: the fast reciprocal is accurate here
  const float2 rA = make_float2(__fdividef(m.x, aA.x), __fdividef(m.y, aA.y));
  const float2 rB = make_float2(__fdividef(m.x, aB.x), __fdividef(m.y, aB.y));
  const float2 rC = make_float2(__fdividef(m.x, aC.x), __fdividef(m.y, aC.y));
  const float2 tA = mul2(v2(0.3f), mul2(rA, rA)), tB = mul2(v2(0.6f), mul2(rB, rB)),
               tC = mul2(v2(0.1f), mul2(rC, rC));
  const float2 num = fma2(tA, cA, fma2(tB, cB, mul2(tC, cC)));
  const float2 den = add2(add2(tA, tB), tC);
  const float2 corr = make_float2(__fdividef(num.x, den.x), __fdividef(num.y, den.y));
  return f2_ + f2v(corr, make_float2(0.f, 0.f));
}

// one lane in FP64
static __device__ __noinline__ f2 weno_fallback64(f2 f0, f2 f1, f2 f2_, f2 f3, f2 f4) {
  return f2_from_double(weno_plus64(f0.to_double(), f1.to_double(), f2_.to_double(),
                                    f3.to_double(), f4.to_double()));
}
__device__ __forceinline__ float f2v_absmax(f2v a) {
  return fmaxf(fabsf(a.hi.x), fabsf(a.hi.y));
}
// unscaled values of any size (a rare path): WV = 0 with weights in float-float, WV = 1 in
// correction form with FP32 weights; in FP64 beyond 1e18
template <int WV>
static __device__ __noinline__ f2v weno_large(f2v f0, f2v f1, f2v f2_, f2v f3, f2v f4) {
  const float mx = fmaxf(fmaxf(fmaxf(f2v_absmax(f0), f2v_absmax(f1)),
                               fmaxf(f2v_absmax(f2_), f2v_absmax(f3))), f2v_absmax(f4));
  if (mx < 1e18f) {
    if constexpr (WV == 1) return weno_plus_f2dv(f0, f1, f2_, f3, f4);
    else return weno_plus_f2v(f0, f1, f2_, f3, f4, 1.f);
  }
  return f2v(weno_fallback64(f0.x(), f1.x(), f2_.x(), f3.x(), f4.x()),
             weno_fallback64(f0.y(), f1.y(), f2_.y(), f3.y(), f4.y()));
}
// the float-float reconstructions of values scaled by kF2Scale
__device__ __forceinline__ f2v weno_pair(f2v f0, f2v f1, f2v f2_, f2v f3, f2v f4) {
  const float mx = fmaxf(fmaxf(fmaxf(f2v_absmax(f0), f2v_absmax(f1)),
                               fmaxf(f2v_absmax(f2_), f2v_absmax(f3))), f2v_absmax(f4));
  if (mx < 1e18f) return weno_plus_f2v(f0, f1, f2_, f3, f4, kF2Scale * kF2Scale);
  const float t = 1.f / kF2Scale;
  return f2v_scale(weno_large<0>(f2v_scale(f0, t), f2v_scale(f1, t), f2v_scale(f2_, t),
                                 f2v_scale(f3, t), f2v_scale(f4, t)), kF2Scale);
}

// split factors of a pair of points, s (u +- alpha)/2 with ha = s alpha/2: lane x the plus side,
// lane y the minus side
__device__ __forceinline__ f2v split_pair(f2 ua, f2 ub, f2 ha, float s) {
  return f2v_scale(f2v(ua, ub), 0.5f * s) + f2v(ha, -ha);
}

// the larger of two magnitudes, NaN if either is
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float f2v_absmax_nan(f2v a) {
  return max_nan(fabsf(a.hi.x), fabsf(a.hi.y));
}
// one advected field: pair k holds c_k (u_k + alpha)/2 and c_{5-k} (u_{5-k} - alpha)/2; h: the
// split factors, scaled for WV = 0.  Returns whether the products are in range: beyond 1e18, or
// past the float range (NaN), the caller takes tracer_large.
template <int WV>
__device__ __forceinline__ bool tracer_face_flux_f2v(const f2v (&h)[5], const f2 (&cv)[6],
                                                     f2& out) {
  constexpr float kS = WV == 1 ? 1.f : kF2Scale;
  f2v a[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) a[k] = f2v(cv[k], cv[5 - k]) * h[k];
  const float mx = max_nan(max_nan(max_nan(f2v_absmax_nan(a[0]), f2v_absmax_nan(a[1])),
                                   max_nan(f2v_absmax_nan(a[2]), f2v_absmax_nan(a[3]))),
                           f2v_absmax_nan(a[4]));
  if (!(mx < 1e18f)) return false;
  f2v r;
  if constexpr (WV == 1) r = weno_plus_f2dv(a[0], a[1], a[2], a[3], a[4]);
  else r = weno_plus_f2v(a[0], a[1], a[2], a[3], a[4], kS * kS);
  out = f2_scale(r.x() + r.y(), 1.f / kS);
  return true;
}

}  // namespace gbmv
