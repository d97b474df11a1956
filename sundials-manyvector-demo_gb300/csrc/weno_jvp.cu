// Derivatives of the WENO flux divergence (the FP64 form of fEuler, src/utilities.cpp:17-253):
//
//   JVP  jv = (d fEuler / d w) dw : forward mode -- the FP64 face flux (weno64.cuh) carried with
//        its directional derivative, then the (linear) divergence.
// The external forcing is constant in w, so it has no derivative.  Kinks (max over the
// stencil of |u| + c, |u|, the positivity guard of sqrt) take the branch the forward pass took.
//
// Bound by the FP64 pipe, so the tangents are written out where a generic dual number would
// spend instructions on constants' zero tangents and on quotients: 36 instructions for the
// tangent of a reconstruction on top of its 33 (weno_tan64).  96^3 x 9: 5330 -> 2139 FP64
// instructions a face.
#include "common.cuh"
#include "weno.cuh"
#include "weno64.cuh"
#include "weno_sweep.cuh"

namespace gbmv {

// a value and its tangent
struct Dual {
  double v, d;
  Dual() = default;
  __device__ Dual(double x, double y) : v(x), d(y) {}
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return Dual(a.v + b.v, a.d + b.d); }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return Dual(a.v - b.v, a.d - b.d); }
__device__ __forceinline__ Dual operator-(Dual a) { return Dual(-a.v, -a.d); }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) {
  return Dual(a.v * b.v, fma(a.v, b.d, a.d * b.v));
}
__device__ __forceinline__ Dual operator*(double a, Dual b) { return Dual(a * b.v, a * b.d); }
__device__ __forceinline__ Dual dfma(Dual a, Dual b, Dual c) {
  return Dual(fma(a.v, b.v, c.v), fma(a.v, b.d, fma(a.d, b.v, c.d)));
}
__device__ __forceinline__ Dual dfma(double a, Dual b, Dual c) {
  return Dual(fma(a, b.v, c.v), fma(a, b.d, c.d));
}
__device__ __forceinline__ Dual drcp(Dual a) {
  const double r = rcp64_any(a.v);
  return Dual(r, -(a.d * (r * r)));
}

// roe64 with tangents
struct RoeDual {
  Dual u, v, w, H, q, c, L00, L01, L02, L03, L04, L30, L31, L40, L41;
};
__device__ __forceinline__ void roe_dual(const Dual (&W)[6][5], const Dual (&ph)[6], double gamma,
                                         RoeDual& R) {
  const double gm = gamma - 1.0;
  const double sL = sqrt0_64(W[2][0].v), sR = sqrt0_64(W[3][0].v);
  const double rL = rcp64_any(sL), rR = rcp64_any(sR);
  const double tL = 0.5 * W[2][0].d * rL, tR = 0.5 * W[3][0].d * rR;  // tangents of the roots
  const Dual iL(rL, -(tL * rL) * rL), iR(rR, -(tR * rR) * rR);
  const Dual is = drcp(Dual(sL + sR, tL + tR));
  R.u = dfma(W[2][1], iL, W[3][1] * iR) * is;
  R.v = dfma(W[2][2], iL, W[3][2] * iR) * is;
  R.w = dfma(W[2][3], iL, W[3][3] * iR) * is;
  R.H = dfma(dfma(2.0, ph[2], W[2][4]), iL, dfma(2.0, ph[3], W[3][4]) * iR) * is;
  R.q = Dual(0.5 * fma(R.u.v, R.u.v, fma(R.v.v, R.v.v, R.w.v * R.w.v)),
             fma(R.u.v, R.u.d, fma(R.v.v, R.v.d, R.w.v * R.w.d)));
  R.c = gm * (R.H - R.q);
  const Dual hc = 0.5 * drcp(R.c), hgc = gm * hc, gq = gm * R.q, gu = gm * R.u;
  R.L00 = hc * (R.u + gq);
  R.L40 = hc * (gq - R.u);
  R.L01 = -dfma(gu, hc, hc);
  R.L41 = hc - gu * hc;
  R.L02 = -(R.v * hgc);
  R.L03 = -(R.w * hgc);
  R.L04 = hgc;
  R.L30 = 2.0 * (hgc * dfma(-2.0, R.q, R.H));
  R.L31 = 2.0 * (R.u * hgc);
}

// fluid_side64 with tangents
template <int SIDE>
__device__ __forceinline__ void fluid_side_dual(const Dual (&W)[6][5], const Dual (&ph)[6],
                                                const Dual (&u)[6], const RoeDual& R,
                                                const Dual (&h)[5], Dual (&ff)[5]) {
  const int j0 = SIDE ? 5 : 0, j1 = SIDE ? 4 : 1, j2 = SIDE ? 3 : 2, j3 = SIDE ? 2 : 3,
            j4 = SIDE ? 1 : 4;
  Dual g[5][5];  // [field]{central, D01, D12, D23, D34}
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    auto point = [&](int q, Dual hq) {
      return m == 1 ? dfma(W[q][1], hq, ph[q])
                    : (m == 4 ? dfma(W[q][4], hq, u[q] * ph[q]) : W[q][m] * hq);
    };
    const Dual f1 = point(j1, h[1]), f2 = point(j2, h[2]), f3 = point(j3, h[3]);
    const Dual r0 = m == 1 ? ph[j0] - f1 : (m == 4 ? dfma(u[j0], ph[j0], -f1) : -f1);
    const Dual r4 = m == 1 ? f3 - ph[j4] : (m == 4 ? dfma(-u[j4], ph[j4], f3) : f3);
    g[m][0] = f2;
    g[m][1] = dfma(W[j0][m], h[0], r0);
    g[m][2] = f1 - f2;
    g[m][3] = f2 - f3;
    g[m][4] = dfma(-W[j4][m], h[4], r4);
  }
  Dual P[5][5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const Dual X = dfma(R.L02, g[2][k], dfma(R.L03, g[3][k], R.L04 * g[4][k]));
    P[k][0] = dfma(R.L00, g[0][k], dfma(R.L01, g[1][k], X));
    P[k][1] = dfma(-R.v, g[0][k], g[2][k]);
    P[k][2] = dfma(-R.w, g[0][k], g[3][k]);
    P[k][3] = dfma(R.L30, g[0][k], dfma(-2.0, X, R.L31 * g[1][k]));
    P[k][4] = dfma(R.L40, g[0][k], dfma(R.L41, g[1][k], X));
  }
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    Weno64 w;
    const double r = weno_diff64(P[0][i].v, P[1][i].v, P[2][i].v, P[3][i].v, P[4][i].v, w);
    ff[i] = Dual(r, weno_tan64(w, P[0][i].d, P[1][i].d, P[2][i].d, P[3][i].d, P[4][i].d));
  }
}

// one tracer's tangent: both sides of c h, the outer points in one difference each
__device__ __forceinline__ double tracer_side_tan(Dual c0, Dual h0, Dual c1, Dual h1, Dual c2,
                                                  Dual h2, Dual c3, Dual h3, Dual c4, Dual h4) {
  const Dual f1 = c1 * h1, f2 = c2 * h2, f3 = c3 * h3;
  const Dual D01 = dfma(c0, h0, -f1), D12 = f1 - f2, D23 = f2 - f3, D34 = dfma(-c4, h4, f3);
  Weno64 w;
  weno_diff64(f2.v, D01.v, D12.v, D23.v, D34.v, w);
  return weno_tan64(w, f2.d, D01.d, D12.d, D23.d, D34.d);
}

// ------------------------------------------------------------------ JVP

// Tangents of the face fluxes, the three directions in one launch.  PRE: the cell primitives
// are read (they live in the fluid part of the result until the divergence), else formed here.
template <int NCHEM, bool PRE>
__global__ void __launch_bounds__(128) face_flux_jvp_kernel(const __grid_constant__ SweepSet S) {
  const int dir = sweep_dir(S);
  const SweepDir& D = S.d[dir];
  const int nblk = (dir == 2 ? (int)gridDim.x : S.d[dir + 1].block0) - D.block0;
  const double gm = S.gamma - 1.0;
  for (long f = (blockIdx.x - D.block0) * (long)blockDim.x + threadIdx.x; f < D.nfaces;
       f += (long)nblk * blockDim.x) {
    long cell[6];
    bool nall[6], nnorm[6];
    stencil_of(S, D, f, false, cell, nall, nnorm);
    Stencil64 T;
    Dual W[6][5], ph[6], u[6];
    double ir[6];
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      double t[5], v1, v2;
      load_point(D.f, cell[l], nall[l], nnorm[l], T.W[l]);
      load_point(D.g, cell[l], nall[l], nnorm[l], t);
      ir[l] = rcp64(T.W[l][0]);
      if (PRE) {
        const double p = __ldg(S.ph + cell[l]), x = __ldg(D.vel[0] + cell[l]);
        T.ph[l] = flip_sign(p, nall[l]);
        T.u[l] = flip_sign(x, nnorm[l]);
        T.hc[l] = __ldg(S.hc + cell[l]);
        v1 = __ldg(D.vel[1] + cell[l]);
        v2 = __ldg(D.vel[2] + cell[l]);
      } else {
        point_prims64(S.gamma, T.W[l][0], T.W[l][1], T.W[l][2], T.W[l][3], T.W[l][4], T.ph[l],
                      T.hc[l]);
        T.u[l] = T.W[l][1] / T.W[l][0];
        v1 = T.W[l][2] / T.W[l][0];
        v2 = T.W[l][3] / T.W[l][0];
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) W[l][v] = Dual(T.W[l][v], t[v]);
      // u = m / rho;  p/2 = (gamma-1)/2 (E - |m|^2 / (2 rho))
      const double x = T.u[l], q = 0.5 * fma(x, x, fma(v1, v1, v2 * v2));
      u[l] = Dual(x, over64(fma(-x, t[0], t[1]), T.W[l][0], ir[l]));
      ph[l] = Dual(T.ph[l], 0.5 * gm *
                   fma(q, t[0], fma(-x, t[1], fma(-v1, t[2], fma(-v2, t[3], t[4])))));
    }
    // half the Lax-Friedrichs speed and its tangent at the point that attains the maximum:
    // (c/2)^2 = gamma (p/2) / (2 rho), so d(c/2) = gamma / (4 rho) (dp/2 - (p/2) drho/rho) / (c/2)
    int am;
    const double ha = half_alpha64(T, &am);
    double su = T.u[0], du = u[0].d, sp = T.ph[0], dp = ph[0].d, sv = T.W[0][0], sr = W[0][0].d,
           si = ir[0], sc = T.hc[0];
#pragma unroll
    for (int l = 1; l < 6; ++l) {
      const bool m = l == am;
      su = m ? T.u[l] : su;
      du = m ? u[l].d : du;
      sp = m ? T.ph[l] : sp;
      dp = m ? ph[l].d : dp;
      sv = m ? T.W[l][0] : sv;
      sr = m ? W[l][0].d : sr;
      si = m ? ir[l] : si;
      sc = m ? T.hc[l] : sc;
    }
    double dha = su < 0.0 ? -0.5 * du : 0.5 * du;
    if (sc > 0.0)
      dha += 0.25 * S.gamma * over64(fma(-over64(sp, sv, si), sr, dp), sv, si) / sc;
    Dual hp[6], hm[6];
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      hp[l] = dfma(0.5, u[l], Dual(ha, dha));
      hm[l] = dfma(0.5, u[l], Dual(-ha, -dha));
    }
    RoeDual R;
    roe_dual(W, ph, S.gamma, R);
    Dual ff[5], fm[5];
    {
      const Dual h[5] = {hp[0], hp[1], hp[2], hp[3], hp[4]};
      fluid_side_dual<0>(W, ph, u, R, h, ff);
    }
    {
      const Dual h[5] = {hm[5], hm[4], hm[3], hm[2], hm[1]};
      fluid_side_dual<1>(W, ph, u, R, h, fm);
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) ff[i] = ff[i] + fm[i];
    const Dual t = ff[0] + ff[4], s = t + ff[3], cd = R.c * (ff[4] - ff[0]);
    const double o[5] = {
        s.d, dfma(R.u, s, cd).d, dfma(R.v, s, ff[1]).d, dfma(R.w, s, ff[2]).d,
        dfma(R.H, t, dfma(R.u, cd, dfma(R.v, ff[1], dfma(R.w, ff[2], R.q * ff[3])))).d};
#pragma unroll
    for (int v = 0; v < 5; ++v) D.F[D.slot[v] * D.nfaces + f] = o[v];
#pragma unroll 1
    for (int c = 0; c < NCHEM; ++c) {
      Dual cv[6];
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        const double x = __ldg(S.chem + c + (long)NCHEM * cell[l]);
        const double dx = __ldg(S.gchem + c + (long)NCHEM * cell[l]);
        cv[l] = Dual(flip_sign(x, nall[l]), flip_sign(dx, nall[l]));
      }
      D.F[(5 + c) * D.nfaces + f] =
          tracer_side_tan(cv[0], hp[0], cv[1], hp[1], cv[2], hp[2], cv[3], hp[3], cv[4], hp[4]) +
          tracer_side_tan(cv[5], hm[5], cv[4], hm[4], cv[3], hm[3], cv[2], hm[2], cv[1], hm[1]);
    }
  }
}

// jv = -sum_d (dF_{d,+} - dF_{d,-}) / d_d
template <int NCHEM>
__global__ void __launch_bounds__(256) divergence_lin_kernel(Grid g, Fields out,
                                                             const double* __restrict__ Fx,
                                                             const double* __restrict__ Fy,
                                                             const double* __restrict__ Fz) {
  const long nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const long nfx = (nx + 1) * ny * nz, nfy = nx * (ny + 1) * nz, nfz = nx * ny * (nz + 1);
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < g.ncell;
       c += (long)gridDim.x * blockDim.x) {
    long i, j, k;
    split3(c, nx, ny, i, j, k);
    const long fx = i + (nx + 1) * (j + ny * k);
    const long fy = i + nx * (j + (ny + 1) * k);
    const long fz = c;
#pragma unroll
    for (int v = 0; v < 5 + NCHEM; ++v) {
      const double div = (Fx[v * nfx + fx + 1] - Fx[v * nfx + fx]) * g.inv_d[0] +
                         (Fy[v * nfy + fy + nx] - Fy[v * nfy + fy]) * g.inv_d[1] +
                         (Fz[v * nfz + fz + nx * ny] - Fz[v * nfz + fz]) * g.inv_d[2];
      double* dst = (v < 5) ? (out.f[v] + c) : (out.f[5] + (v - 5) + (long)NCHEM * c);
      *dst = -div;
    }
  }
}

// ------------------------------------------------------------------ launcher

template <int NCHEM>
static int jvp_t(const Grid& g, const Fields& w, const Fields& dw, const Fields& out,
                 double* scratch, cudaStream_t s) {
  long nf[3];
  face_counts(g, nf);
  double* F[3] = {scratch, scratch + (long)(5 + NCHEM) * nf[0],
                  scratch + (long)(5 + NCHEM) * (nf[0] + nf[1])};
  ProfScope ps("jvp", s);
  // the primitives live in the fluid part of the result, which the divergence writes last,
  // unless the call is in place
  const bool pre = !fields_overlap(g, w, out) && !fields_overlap(g, dw, out);
  const int t = spread_threads(nf[0] + nf[1] + nf[2], 128);
  SweepSet S;
  const int b = sweep_set(g, w, F, 1, t, (long)kSM * 16, S);
  sweep_second(S, dw);
  if (pre) {
    double* const p[5] = {out.f[0], out.f[1], out.f[2], out.f[3], out.f[4]};
    const int rc = prims64(g, w, p, nullptr, s);
    if (rc) return rc;
    const double* const u[3] = {p[1], p[2], p[3]};
    sweep_prims(S, p[0], u, p[4]);
    face_flux_jvp_kernel<NCHEM, true><<<b, t, 0, s>>>(S);
  } else {
    face_flux_jvp_kernel<NCHEM, false><<<b, t, 0, s>>>(S);
  }
  GBMV_LAUNCH_CHECK("face_flux_jvp_kernel");
  divergence_lin_kernel<NCHEM><<<sweep_blocks(g.ncell, 256), 256, 0, s>>>(g, out, F[0], F[1], F[2]);
  GBMV_LAUNCH_CHECK("divergence_lin_kernel");
  return GBMV_OK;
}

int feuler_jvp(const Grid& g, const Fields& w, const Fields& dw, const Fields& out,
               double* scratch, cudaStream_t s) {
  switch (g.nchem) {
    case 0: return jvp_t<0>(g, w, dw, out, scratch, s);
    case 2: return jvp_t<2>(g, w, dw, out, scratch, s);
    case 4: return jvp_t<4>(g, w, dw, out, scratch, s);
    case 6: return jvp_t<6>(g, w, dw, out, scratch, s);
    case 10: return jvp_t<10>(g, w, dw, out, scratch, s);
    default: return GBMV_EUNSUPPORTED;
  }
}

}  // namespace gbmv
