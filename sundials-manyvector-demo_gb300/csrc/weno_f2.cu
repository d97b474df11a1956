// Float-float WENO flux divergence: the per-cell primitive pass, the fluid sweep and the entry
// point that picks the tracers' weights (weno_f2.cuh).
#include "weno_f2.cuh"

namespace gbmv {

// Register budgets of the sweeps (128-thread blocks per SM; the same bits whatever they are; timed
// with un-normalised projections: 2.51 ms is 2.54 with the normalised ones).
// Fluid, 128^3 x 15 GBMV_MIXED_FAST RHS at 2 / 3 / 4 blocks: 2.61 / 2.51 / 2.57 ms.  Beside the
// chemistry Newton on a second stream (255 registers a thread) 5 leave the Newton's warps room
// (Grid::sweep_shared).  Tracers: FP32 weights 5 / 6 / 7 / 8: 2.53 / 2.51 / 2.51 / 2.53
// ms; float-float weights 4 / 5 / 6 (128^3 x 9 GBMV_MIXED): 2.34 / 2.32 / 2.32 ms.
constexpr int kF2MinB = 3;
constexpr int kF2SharedMinB = 5;
constexpr int kTracerFastMinB = 6;
constexpr int kTracerMinB = 5;

__global__ void __launch_bounds__(256) prims_f2_kernel(Grid g, Fields w, float2* __restrict__ Q2,
                                                       const double* __restrict__ tscale,
                                                       int* __restrict__ status) {
  const long n = g.ncell;
  int bad = 0;
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n;
       c += (long)gridDim.x * blockDim.x) {
    const double rho = w.f[0][c], mx = w.f[1][c], my = w.f[2][c], mz = w.f[3][c], et = w.f[4][c];
    // one FP64 division per cell: the primitives are multiplied by 1/rho (each within an ulp
    // of the reference's quotients, far inside the float-float representation error)
    const double ir = 1.0 / rho;
    const double p = (g.gamma - 1.0) * (et - (mx * mx + my * my + mz * mz) * 0.5 * ir);
    // legal_state (src/euler3D.hpp:1398-1414) on this pressure: it differs from the quotient
    // form only in the last bit, so only a state with p within rounding of zero can flag
    // differently from the FP64 form
    bad |= (!(rho > 0.0) ? 1 : 0) | (!(et > 0.0) ? 2 : 0) | (!(p > 0.0) ? 4 : 0);
    double q[kQ2Base] = {rho, mx, my, mz, et, p, mx * ir, my * ir, mz * ir,
                         sqrt0_64(g.gamma * p * ir)};
#pragma unroll
    for (int k = 0; k < kQ2Base; ++k) {
      const f2 v = f2_split(q[k]);
      Q2[k * n + c] = make_float2(v.hi, v.lo);
    }
    for (int v = 0; v < g.nchem; ++v) {
      // tscale: the chemistry component arrives in scaled units (x = chem * scale)
      const long e = v + (long)g.nchem * c;
      const f2 x = f2_split(tscale ? w.f[5][e] * tscale[e] : w.f[5][e]);
      Q2[(kQ2Base + v) * n + c] = make_float2(x.hi, x.lo);
    }
  }
  bad = __reduce_or_sync(0xffffffffu, bad);
  if (bad && (threadIdx.x & 31) == 0) atomicOr(status, bad);
}

int prims_f2(const Grid& g, const Fields& w, float2* q2, const double* tscale, int* d_status,
             cudaStream_t s) {
  ProfScope ps("prims", s);
  prims_f2_kernel<<<sweep_blocks(g.ncell, 256), 256, 0, s>>>(g, w, q2, tscale, d_status);
  GBMV_LAUNCH_CHECK("prims_f2_kernel");
  return GBMV_OK;
}

// A face of the fluid sweep in FP64, exactly the FP64 form's arithmetic: fluxes, and half the
// Lax-Friedrichs speed.
static __device__ __noinline__ void fluid_face_64(const SweepSet& S, const SweepDir& D, long f,
                                                  f2 (&out)[5], f2& ha) {
  long cell[6];
  bool nall[6], nnorm[6];
  stencil_of(S, D, f, false, cell, nall, nnorm);
  Stencil64 T;
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    load_point(D.f, cell[l], nall[l], nnorm[l], T.W[l]);
    point_prims64(S.gamma, T.W[l][0], T.W[l][1], T.W[l][2], T.W[l][3], T.W[l][4], T.ph[l],
                  T.hc[l]);
    T.u[l] = T.W[l][1] / T.W[l][0];
  }
  Split64 H;
  double o[5];
  fluid_face_flux64<false>(T, S.gamma, H, o);
#pragma unroll
  for (int v = 0; v < 5; ++v) out[v] = f2_from_double(o[v]);
  ha = f2_from_double(half_alpha64(T));
}

// Fluid face fluxes of the three directions; with tracers, half the Lax-Friedrichs speed is left
// in the first tracer's flux for the tracer sweep.  MINB: register budget (residency target in
// 128-thread blocks; the same bits whatever it is).
template <int MINB>
__global__ void __launch_bounds__(128, MINB)
    fluid_flux_f2_kernel(const __grid_constant__ SweepSet S, const float2* __restrict__ Q2, long n,
                         int nchem) {
  const SweepDir& D = S.d[blockIdx.x % 3];
  float2* const F = reinterpret_cast<float2*>(D.F);
  for (long f = (blockIdx.x / 3) * (long)blockDim.x + threadIdx.x; f < D.nfaces;
       f += (gridDim.x / 3) * (long)blockDim.x) {
    StencilF2 T;
    stencil_f2(S, D, f, T);
    const f2 gm = f2_from_double(S.gamma - 1.0);
    // a fluid value of point l in face order with its ghost sign (homogeneous Dirichlet negates
    // every conserved field, so p too; reflecting the normal momentum and velocity)
    const int src[5] = {0, D.slot[1], D.slot[2], D.slot[3], 4};
    auto val = [&](int v, int l) {
      f2 q = q2_load(Q2, n, src[v], T.cell[l]);
      if (((T.nall ^ (v == 1 ? T.nnorm : 0u)) >> l) & 1u) q = -q;
      return q;
    };
    auto pressure = [&](int l) {
      const f2 q = q2_load(Q2, n, 5, T.cell[l]);
      return (T.nall >> l) & 1u ? -q : q;
    };
    auto velocity = [&](int l) {
      const f2 q = q2_load(Q2, n, 6 + D.dir, T.cell[l]);
      return (T.nnorm >> l) & 1u ? -q : q;
    };
    // Lax-Friedrichs speed (src/utilities.cpp:368-380)
    f2 alpha(0.0);
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      const f2 s = f2_fabs(velocity(l)) + q2_load(Q2, n, 9, T.cell[l]);
      alpha = (alpha < s) ? s : alpha;
    }
    f2 ha = f2_scale(alpha, 0.5f);
    // Roe average (src/utilities.cpp:298-304) and the left eigenvector rows (:342-364)
    f2 u, v, w, H, q, c, L00, L01, L02, L03, L04, L30, L31, L40, L41;
    {
      const f2 one(1.0);
      const f2 sL = f2_sqrt0(val(0, 2)), sR = f2_sqrt0(val(0, 3));
      const f2 iL = one / sL, iR = one / sR, is = one / (sL + sR);
      u = (val(1, 2) * iL + val(1, 3) * iR) * is;
      v = (val(2, 2) * iL + val(2, 3) * iR) * is;
      w = (val(3, 2) * iL + val(3, 3) * iR) * is;
      H = ((pressure(2) + val(4, 2)) * iL + (pressure(3) + val(4, 3)) * iR) * is;
      q = f2_scale(u * u + v * v + w * w, 0.5f);
      c = gm * (H - q);  // the reference's "csnd" (src/utilities.cpp:309)
      const f2 hc = f2_scale(one / c, 0.5f), hgc = gm * hc, gc = f2_scale(hgc, 2.f), gq = gm * q,
               gu = gm * u;
      L00 = hc * (u + gq);
      L40 = hc * (gq - u);
      L01 = -(hc * (gu + one));
      L41 = -(hc * (gu - one));
      L02 = -(v * hgc);
      L03 = -(w * hgc);
      L04 = hgc;
      L30 = gc * (H - f2_scale(q, 2.f));
      L31 = u * gc;
    }
    bool ok = true;
    const f2 has = f2_scale(ha, kF2Scale);
    f2v P[5][5];  // [pair][characteristic component], times kF2Scale
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int a = k, b = 5 - k;
      f2v Wj[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        Wj[m] = f2v(val(m, a), val(m, b));
        ok = ok && f2v_absmax(Wj[m]) < 1e15f;
      }
      const f2v pj = f2v_scale(f2v(pressure(a), pressure(b)), 0.5f * kF2Scale);
      ok = ok && fminf(Wj[0].hi.x, Wj[0].hi.y) > 0.f && f2v_absmax(pj) < 5e14f * kF2Scale;
      const f2 ua = velocity(a), ub = velocity(b);
      const f2v h = split_pair(ua, ub, has, kF2Scale), uj(ua, ub);
      const f2v f0 = Wj[0] * h, f1 = f2v_fma(Wj[1], h, pj), f2_ = Wj[2] * h, f3 = Wj[3] * h,
                f4 = f2v_fma(uj, pj, Wj[4] * h);
      ok = ok && f2v_absmax(f4) < 1e30f;  // the energy flux, the largest: no overflow below
      // (every product is normalised: left un-normalised the sums took 1 % less time, 256^3 x 15
      // 19.84 and 20.02 ms, and single fields' largest errors were up to 1.5 times the normalised ones)
      const f2v X = f2v_fma(f2v(L04), f4, f2v_fma(f2v(L03), f3, f2v(L02) * f2_));
      P[k][0] = f2v_fma(f2v(L01), f1, f2v_fma(f2v(L00), f0, X));
      P[k][1] = f2v_fma(f2v(-v), f0, f2_);
      P[k][2] = f2v_fma(f2v(-w), f0, f3);
      P[k][3] = f2v_fma(f2v(L31), f1, f2v_fma(f2v(L30), f0, f2v_scale(X, -2.f)));
      P[k][4] = f2v_fma(f2v(L41), f1, f2v_fma(f2v(L40), f0, X));
    }
    f2 o[5];
    if (ok) {
      f2 ff[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const f2v r = weno_pair(P[0][i], P[1][i], P[2][i], P[3][i], P[4][i]);
        ff[i] = f2_scale(r.x() + r.y(), 1.f / kF2Scale);
      }
      // right eigenvector columns (src/utilities.cpp:318-340)
      const f2 t = ff[0] + ff[4], s = t + ff[3], cd = c * (ff[4] - ff[0]);
      o[0] = s;
      o[1] = u * s + cd;
      o[2] = v * s + ff[1];
      o[3] = w * s + ff[2];
      o[4] = H * t + (u * cd + (v * ff[1] + (w * ff[2] + q * ff[3])));
    } else {
      fluid_face_64(S, D, f, o, ha);
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) F[D.slot[m] * D.nfaces + f] = make_float2(o[m].hi, o[m].lo);
    if (nchem) F[5 * D.nfaces + f] = make_float2(ha.hi, ha.lo);
  }
}

// The reconstructions of a tracer whose split fluxes pass the range of the scaled arithmetic, from
// the start and without the scale (ha: half the Lax-Friedrichs speed).
template <int WV>
static __device__ __noinline__ f2 tracer_large(const SweepSet& S, const SweepDir& D, long f,
                                               const float2* __restrict__ Q2, long n, int c,
                                               f2 ha) {
  StencilF2 T;
  stencil_f2(S, D, f, T);
  f2 u[6], v[6];
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    u[l] = q2_load(Q2, n, 6 + D.dir, T.cell[l]);
    v[l] = q2_load(Q2, n, kQ2Base + c, T.cell[l]);
    if ((T.nnorm >> l) & 1u) u[l] = -u[l];
    if ((T.nall >> l) & 1u) v[l] = -v[l];
  }
  f2v a[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) a[k] = f2v(v[k], v[5 - k]) * split_pair(u[k], u[5 - k], ha, 1.f);
  const f2v r = weno_large<WV>(a[0], a[1], a[2], a[3], a[4]);
  return r.x() + r.y();
}

// Tracer face fluxes: one thread a face, its tracers one after the other; reads half the
// Lax-Friedrichs speed that the fluid sweep left in the first tracer's flux.
template <int WV>
__global__ void __launch_bounds__(128, WV == 1 ? kTracerFastMinB : kTracerMinB)
    tracer_flux_f2_kernel(const __grid_constant__ SweepSet S, const float2* __restrict__ Q2,
                          long n, int nchem) {
  const SweepDir& D = S.d[blockIdx.x % 3];
  float2* const F = reinterpret_cast<float2*>(D.F);
  for (long f = (blockIdx.x / 3) * (long)blockDim.x + threadIdx.x; f < D.nfaces;
       f += (gridDim.x / 3) * (long)blockDim.x) {
    StencilF2 T;
    stencil_f2(S, D, f, T);
    f2v h[5];
    const float2 t = F[5 * D.nfaces + f];
    {
      const float sc = WV == 1 ? 1.f : kF2Scale;
      const f2 ha(sc * t.x, sc * t.y);
      f2 u[6];
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        u[l] = q2_load(Q2, n, 6 + D.dir, T.cell[l]);
        if ((T.nnorm >> l) & 1u) u[l] = -u[l];
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) h[k] = split_pair(u[k], u[5 - k], ha, sc);
    }
#pragma unroll 1
    for (int c = 0; c < nchem; ++c) {
      f2 cv[6];
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        cv[l] = q2_load(Q2, n, kQ2Base + c, T.cell[l]);
        if ((T.nall >> l) & 1u) cv[l] = -cv[l];
      }
      f2 r;
      if (!tracer_face_flux_f2v<WV>(h, cv, r)) r = tracer_large<WV>(S, D, f, Q2, n, c, f2(t.x, t.y));
      F[(5 + c) * D.nfaces + f] = make_float2(r.hi, r.lo);
    }
  }
}

size_t feuler_f2_prims_floats(const Grid& g) { return (size_t)2 * (kQ2Base + g.nchem) * g.ncell; }

int feuler_f2(const Grid& g, const Fields& w, const Fields& wdot, const ForceTerm& G,
              double* scratch, float* prims, const double* tscale, int* d_status,
              cudaStream_t s, int fast_weights) {
  float2* const q2 = reinterpret_cast<float2*>(prims);
  long nf[3];
  face_counts(g, nf);
  const long nv = 5 + g.nchem;
  double* const F[3] = {scratch, scratch + nv * nf[0], scratch + nv * (nf[0] + nf[1])};
  float2* const F2[3] = {reinterpret_cast<float2*>(F[0]), reinterpret_cast<float2*>(F[1]),
                         reinterpret_cast<float2*>(F[2])};
  int rc = prims_f2(g, w, q2, tscale, d_status, s);
  if (rc != GBMV_OK) return rc;
  {
    ProfScope ps("face_flux", s);
    const int t = sweep_threads(g, nf[0] + nf[1] + nf[2], 128);
    SweepSet S;
    sweep_set(g, w, F, 1, t, 1L << 30, S);
    // One face a thread and the directions in turn, block by block: the three read the same cells
    // at about the same time, from L2.  (A grid of 16 blocks per SM and direction, each walking
    // over its direction, one direction after the other: 128^3 x 15 GBMV_MIXED_FAST 2622 -> 2504
    // us, 256^3 21.97 -> 19.92 ms, 160 x 150 x 140 x 7 3242 -> 2950 us, at 10^5 cells the same.
    // The kernels' loops then run once; a plain test in their place compiles to 1.5 % more.)
    const long most = nf[0] > nf[1] ? nf[0] : nf[1];
    const int b = (int)(3 * (((most > nf[2] ? most : nf[2]) + t - 1) / t));
    if (fast_weights && g.sweep_shared)
      fluid_flux_f2_kernel<kF2SharedMinB><<<b, t, 0, s>>>(S, q2, g.ncell, g.nchem);
    else
      fluid_flux_f2_kernel<kF2MinB><<<b, t, 0, s>>>(S, q2, g.ncell, g.nchem);
    GBMV_LAUNCH_CHECK("fluid_flux_f2_kernel");
    if (g.nchem) {
      if (fast_weights) tracer_flux_f2_kernel<1><<<b, t, 0, s>>>(S, q2, g.ncell, g.nchem);
      else tracer_flux_f2_kernel<0><<<b, t, 0, s>>>(S, q2, g.ncell, g.nchem);
      GBMV_LAUNCH_CHECK("tracer_flux_f2_kernel");
    }
  }
  return divergence_f2(g, wdot, F2, G, s);
}

}  // namespace gbmv
