// Derivatives of the WENO flux divergence (the FP64 form of fEuler, src/utilities.cpp:17-253):
//   VJP  u = (d fEuler / d w)^T v : reverse mode, hand-written.  Per face: the face cotangent
//        from the divergence, cF = (v_{i} - v_{i-1}) / dx along the face normal, then the
//        adjoint of the characteristic face flux (Roe average, eigenvectors, Lax-Friedrichs
//        splitting, WENO5 weights, back-projection) gives the cotangents of the six stencil
//        points, with the direction swap and the ghost signs undone; these are stored per face
//        and stencil slot and a per-cell gather (inverse of the ghost rule, so no atomics and a
//        deterministic result) sums them into u.
// The external forcing is constant in w, so it has no derivative.  Kinks (max over the
// stencil of |u| + c, |u|, the positivity guard of sqrt) take the branch the forward pass took.
//
// Bound by the FP64 pipe.  The adjoint of a reconstruction works on the neighbour differences
// and takes the forward weights' products (weno_adj64: 40 instructions after the forward 33; the
// adjoint of the literal formula took ~250 with its seven divisions), the primitives come from
// a cell pass, and each point's reciprocal density is formed once.  96^3 x 9: 6120 -> 2350
// FP64 instructions a face.
#include "common.cuh"
#include "weno.cuh"
#include "weno64.cuh"
#include "weno_sweep.cuh"

namespace gbmv {

// ------------------------------------------------------------------ VJP

// the five split fluxes of a point, as fluid_side64 forms them
__device__ __forceinline__ void split_point64(const Stencil64& S, int j, double h,
                                              double (&f)[5]) {
  f[0] = S.W[j][0] * h;
  f[1] = fma(S.W[j][1], h, S.ph[j]);
  f[2] = S.W[j][2] * h;
  f[3] = S.W[j][3] * h;
  f[4] = fma(S.W[j][4], h, S.u[j] * S.ph[j]);
}

// Cotangents gathered over the face: of the Roe values and eigenvector entries, of the points'
// state, half pressure, velocity and of half the Lax-Friedrichs speed.
struct Adj64 {
  double W[6][5], ph[6], u[6], ha;
  double v, w;
  double L00, L01, L02, L03, L04, L30, L31, L40, L41;
};

// characteristic values of one side, points in upwind order as fluid_side64
template <int SIDE>
__device__ __forceinline__ void fluid_side_project(const Stencil64& S, const Roe64& R,
                                                   const double (&h)[5], double (&P)[5][5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    double f[5];
    split_point64(S, SIDE ? 5 - k : k, h[k], f);
    const double X = fma(R.L02, f[2], fma(R.L03, f[3], R.L04 * f[4]));
    P[k][0] = fma(R.L00, f[0], fma(R.L01, f[1], X));
    P[k][1] = fma(-R.v, f[0], f[2]);
    P[k][2] = fma(-R.w, f[0], f[3]);
    P[k][3] = fma(R.L30, f[0], fma(-2.0, X, R.L31 * f[1]));
    P[k][4] = fma(R.L40, f[0], fma(R.L41, f[1], X));
  }
}

// The forward reconstruction of component i and, in place of its five points, their cotangents
__device__ __forceinline__ double weno_fwd_adj(double (&P)[5][5], int i, double rb) {
  Weno64 w;
  const double r = weno_diff64(P[2][i], P[0][i] - P[1][i], P[1][i] - P[2][i], P[2][i] - P[3][i],
                               P[3][i] - P[4][i], w);
  double b[5];
  weno_adj64(w, rb, b);
#pragma unroll
  for (int k = 0; k < 5; ++k) P[k][i] = b[k];
  return r;
}

// One side of the fluid part: from the cotangents ffb of its reconstructions, their values into
// ff and the adjoint of projection and splitting into B.
template <int SIDE>
__device__ __forceinline__ void fluid_side_adj(const Stencil64& S, const Roe64& R,
                                               const double (&h)[5], const double (&ffb)[5],
                                               double (&ff)[5], Adj64& B) {
  double P[5][5];
  fluid_side_project<SIDE>(S, R, h, P);
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const double r = weno_fwd_adj(P, i, ffb[i]);
    ff[i] = SIDE ? ff[i] + r : r;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int j = SIDE ? 5 - k : k;
    const double(&b)[5] = P[k];
    double f[5], fb[5];
    split_point64(S, j, h[k], f);
    const double Xb = fma(-2.0, b[3], b[0] + b[4]);
    B.L00 = fma(b[0], f[0], B.L00);
    B.L01 = fma(b[0], f[1], B.L01);
    B.L02 = fma(Xb, f[2], B.L02);
    B.L03 = fma(Xb, f[3], B.L03);
    B.L04 = fma(Xb, f[4], B.L04);
    B.L30 = fma(b[3], f[0], B.L30);
    B.L31 = fma(b[3], f[1], B.L31);
    B.L40 = fma(b[4], f[0], B.L40);
    B.L41 = fma(b[4], f[1], B.L41);
    B.v = fma(-b[1], f[0], B.v);
    B.w = fma(-b[2], f[0], B.w);
    fb[0] = fma(R.L00, b[0], fma(R.L40, b[4], fma(R.L30, b[3], fma(-R.v, b[1], -R.w * b[2]))));
    fb[1] = fma(R.L01, b[0], fma(R.L41, b[4], R.L31 * b[3]));
    fb[2] = fma(R.L02, Xb, b[1]);
    fb[3] = fma(R.L03, Xb, b[2]);
    fb[4] = R.L04 * Xb;
    double hb = 0.0;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      B.W[j][m] = fma(h[k], fb[m], B.W[j][m]);
      hb = m ? fma(S.W[j][m], fb[m], hb) : S.W[j][0] * fb[0];
    }
    B.ph[j] += fma(S.u[j], fb[4], fb[1]);
    B.u[j] = fma(S.ph[j], fb[4], fma(0.5, hb, B.u[j]));
    B.ha = SIDE ? B.ha - hb : B.ha + hb;
  }
}

// one side of a tracer: cotangents of its values and of the split factors
__device__ __forceinline__ void tracer_side_adj(const double (&c)[5], const double (&h)[5],
                                                double rb, double (&cb)[5], double (&hb)[5]) {
  Weno64 w;
  weno_prod64(c[0], h[0], c[1], h[1], c[2], h[2], c[3], h[3], c[4], h[4], w);
  double b[5];
  weno_adj64(w, rb, b);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    cb[k] = b[k] * h[k];
    hb[k] = fma(b[k], c[k], hb[k]);
  }
}

// Face cotangents -> per-face stencil cotangents A[(l * NVAR + v) * nfaces + f] (original
// field order, ghost signs applied, so each entry belongs to the source cell of slot l), for the
// one direction the launch covers.  S.d[dir].g: the cotangent ManyVector in face order.
template <int NCHEM>
__global__ void __launch_bounds__(128) face_flux_vjp_kernel(const __grid_constant__ SweepSet S,
                                                            int dir, double inv_d,
                                                            double* __restrict__ A) {
  constexpr int NV = 5 + NCHEM;
  const SweepDir& D = S.d[dir];
  const long nfaces = D.nfaces;
  const double gm = S.gamma - 1.0;
  for (long f = blockIdx.x * (long)blockDim.x + threadIdx.x; f < nfaces;
       f += (long)gridDim.x * blockDim.x) {
    long cell[6];
    bool nall[6], nnorm[6];
    stencil_of(S, D, f, false, cell, nall, nnorm);
    // face cotangent: + v_i / d for the cell above (i < n), - v_{i-1} / d for the one below
    long i0, j0, k0;
    split3(f, D.ex, D.ey, i0, j0, k0);
    const long id = dir == 0 ? i0 : (dir == 1 ? j0 : k0);
    const long cup = i0 + S.nx * (j0 + S.ny * k0);  // valid when id < n
    const long cdn = cup - D.stride;
    double ob[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      double a = 0.0;
      if (id < D.n) a = D.g[v][cup];
      if (id >= 1) a -= D.g[v][cdn];
      ob[v] = a * inv_d;
    }
    Stencil64 T;
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      load_point(D.f, cell[l], nall[l], nnorm[l], T.W[l]);
      const double p = __ldg(S.ph + cell[l]), x = __ldg(D.vel[0] + cell[l]);
      T.ph[l] = flip_sign(p, nall[l]);
      T.u[l] = flip_sign(x, nnorm[l]);
      T.hc[l] = __ldg(S.hc + cell[l]);
    }
    int am;
    const double ha = half_alpha64(T, &am);
    double hp[5], hm[5];  // both sides in upwind order (hm[k] belongs to point 5 - k)
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      hp[k] = fma(0.5, T.u[k], ha);
      hm[k] = fma(0.5, T.u[5 - k], -ha);
    }
    // tracers first: their cotangents of the split factors join the fluid part's
    double hpb[5] = {0, 0, 0, 0, 0}, hmb[5] = {0, 0, 0, 0, 0};
#pragma unroll 1
    for (int c = 0; c < NCHEM; ++c) {
      double rb = 0.0;
      if (id < D.n) rb = S.gchem[c + (long)NCHEM * cup];
      if (id >= 1) rb -= S.gchem[c + (long)NCHEM * cdn];
      rb *= inv_d;
      double cv[6];
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        cv[l] = flip_sign(__ldg(S.chem + c + (long)NCHEM * cell[l]), nall[l]);
      }
      double pb[5], mb[5];
      {
        const double a[5] = {cv[0], cv[1], cv[2], cv[3], cv[4]};
        tracer_side_adj(a, hp, rb, pb, hpb);
      }
      {
        const double a[5] = {cv[5], cv[4], cv[3], cv[2], cv[1]};
        tracer_side_adj(a, hm, rb, mb, hmb);
      }
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        const double b = l == 0 ? pb[0] : (l == 5 ? mb[0] : pb[l] + mb[5 - l]);
        A[((long)l * NV + 5 + c) * nfaces + f] = flip_sign(b, nall[l]);
      }
    }
    Adj64 B;
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      B.ph[l] = B.u[l] = 0.0;
#pragma unroll
      for (int m = 0; m < 5; ++m) B.W[l][m] = 0.0;
    }
    B.ha = 0.0;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      B.u[k] = fma(0.5, hpb[k], B.u[k]);
      B.u[5 - k] = fma(0.5, hmb[k], B.u[5 - k]);
      B.ha += hpb[k] - hmb[k];
    }
    Roe64 R;
    roe64(T, S.gamma, R);
    const double u = R.u, v = R.v, w = R.w, c = R.c;
    // back-projection (fluid_back64): s = ff0 + ff3 + ff4, t = ff0 + ff4, cd = c (ff4 - ff0)
    const double sb = fma(ob[1], u, fma(ob[2], v, fma(ob[3], w, ob[0])));
    const double tb = sb + ob[4] * R.H, cdb = fma(ob[4], u, ob[1]), db = cdb * c;
    const double ffb[5] = {tb - db, fma(ob[4], v, ob[2]), fma(ob[4], w, ob[3]),
                           fma(ob[4], R.q, sb), tb + db};
    B.v = B.w = B.L00 = B.L01 = B.L02 = B.L03 = B.L04 = B.L30 = B.L31 = B.L40 = B.L41 = 0.0;
    double ff[5];
    fluid_side_adj<0>(T, R, hp, ffb, ff, B);
    fluid_side_adj<1>(T, R, hm, ffb, ff, B);
    const double t = ff[0] + ff[4], s = t + ff[3], d = ff[4] - ff[0];
    double ub = fma(ob[1], s, ob[4] * (c * d)), vb = B.v + fma(ob[2], s, ob[4] * ff[1]),
           wb = B.w + fma(ob[3], s, ob[4] * ff[2]), Hb = ob[4] * t, qb = ob[4] * ff[3],
           cb = cdb * d;
    // left eigenvector entries; hc = 1/(2c), hgc = gm hc, gc = 2 hgc
    const double hc = 0.5 * rcp64_any(c), hgc = gm * hc, gq = gm * R.q, gu = gm * u;
    double hcb = fma(B.L00, u + gq, fma(B.L40, gq - u, -fma(B.L01, gu + 1.0, B.L41 * (gu - 1.0))));
    ub = fma(hc, (B.L00 - B.L40) - gm * (B.L01 + B.L41), ub);
    qb = fma(hgc, B.L00 + B.L40, qb);
    double hgcb = B.L04 - fma(v, B.L02, w * B.L03);
    vb = fma(-hgc, B.L02, vb);
    wb = fma(-hgc, B.L03, wb);
    hgcb = fma(2.0, fma(B.L30, fma(-2.0, R.q, R.H), B.L31 * u), hgcb);
    Hb = fma(2.0 * hgc, B.L30, Hb);
    qb = fma(-4.0 * hgc, B.L30, qb);
    ub = fma(2.0 * hgc, B.L31, ub);
    hcb = fma(gm, hgcb, hcb);
    cb = fma(-2.0 * (hc * hc), hcb, cb);  // d(1/(2c)) = -2 hc^2 dc
    // c = gm (H - q),  q = (u^2 + v^2 + w^2) / 2
    Hb = fma(gm, cb, Hb);
    qb = fma(-gm, cb, qb);
    ub = fma(u, qb, ub);
    vb = fma(v, qb, vb);
    wb = fma(w, qb, wb);
    // Roe averages X = (a iL + b iR) is, iL = 1/sqrt(rhoL), is = 1/(sL + sR)
    {
      const double sL = sqrt0_64(T.W[2][0]), sR = sqrt0_64(T.W[3][0]);
      const double iL = rcp64_any(sL), iR = rcp64_any(sR), is = rcp64_any(__dadd_rn(sL, sR));
      const double eL = fma(2.0, T.ph[2], T.W[2][4]), eR = fma(2.0, T.ph[3], T.W[3][4]);
      const double xu = ub * is, xv = vb * is, xw = wb * is, xH = Hb * is;
      B.W[2][1] = fma(xu, iL, B.W[2][1]);
      B.W[3][1] = fma(xu, iR, B.W[3][1]);
      B.W[2][2] = fma(xv, iL, B.W[2][2]);
      B.W[3][2] = fma(xv, iR, B.W[3][2]);
      B.W[2][3] = fma(xw, iL, B.W[2][3]);
      B.W[3][3] = fma(xw, iR, B.W[3][3]);
      B.W[2][4] = fma(xH, iL, B.W[2][4]);
      B.W[3][4] = fma(xH, iR, B.W[3][4]);
      B.ph[2] = fma(2.0 * xH, iL, B.ph[2]);
      B.ph[3] = fma(2.0 * xH, iR, B.ph[3]);
      const double iLb = fma(xu, T.W[2][1], fma(xv, T.W[2][2], fma(xw, T.W[2][3], xH * eL)));
      const double iRb = fma(xu, T.W[3][1], fma(xv, T.W[3][2], fma(xw, T.W[3][3], xH * eR)));
      // every X carries the factor is: is b = sum X b X / is, d(is) = -is^2 (dsL + dsR)
      const double sb2 = -is * fma(ub, u, fma(vb, v, fma(wb, w, Hb * R.H)));
      // d iL = -iL^2 dsL, dsL = drho iL / 2
      if (T.W[2][0] > 0.0)
        B.W[2][0] = fma(0.5 * iL, fma(-iL, iL * iLb, sb2), B.W[2][0]);
      if (T.W[3][0] > 0.0)
        B.W[3][0] = fma(0.5 * iR, fma(-iR, iR * iRb, sb2), B.W[3][0]);
    }
    // half the Lax-Friedrichs speed at its point: ha = |u|/2 + c/2,
    // d(c/2) = gamma / (4 rho) (d(p/2) - (p/2) drho / rho) / (c/2)
    {
      double sr = T.W[0][0], sp = T.ph[0], sc = T.hc[0], su = T.u[0];
#pragma unroll
      for (int l = 1; l < 6; ++l) {
        const bool m = l == am;
        sr = m ? T.W[l][0] : sr;
        sp = m ? T.ph[l] : sp;
        sc = m ? T.hc[l] : sc;
        su = m ? T.u[l] : su;
      }
      const double uadd = su < 0.0 ? -0.5 * B.ha : 0.5 * B.ha;
      double padd = 0.0, radd = 0.0;
      if (sc > 0.0) {
        const double ir = rcp64(sr);
        padd = 0.25 * S.gamma * over64(B.ha, sr, ir) / sc;
        radd = -over64(padd * sp, sr, ir);
      }
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        const bool m = l == am;
        B.u[l] += m ? uadd : 0.0;
        B.ph[l] += m ? padd : 0.0;
        B.W[l][0] += m ? radd : 0.0;
      }
    }
    // points' primitives: u = m / rho, p/2 = gm/2 (E - |m|^2 / (2 rho))
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      const double ir = rcp64(T.W[l][0]), x = T.u[l], v1 = __ldg(D.vel[1] + cell[l]),
                   v2 = __ldg(D.vel[2] + cell[l]);
      const double k = 0.5 * gm * B.ph[l], m = over64(B.u[l], T.W[l][0], ir);
      double q[5];
      q[0] = fma(k, 0.5 * fma(x, x, fma(v1, v1, v2 * v2)), fma(-m, x, B.W[l][0]));
      q[1] = fma(-k, x, B.W[l][1] + m);
      q[2] = fma(-k, v1, B.W[l][2]);
      q[3] = fma(-k, v2, B.W[l][3]);
      q[4] = B.W[l][4] + k;
#pragma unroll
      for (int e = 0; e < 5; ++e)
        A[((long)l * NV + D.slot[e]) * nfaces + f] =
            flip_sign(q[e], nall[l] != (e == 1 && nnorm[l]));
    }
  }
}

// u (+)= sum over the (face, slot) pairs whose source cell is c of A[(slot, v), face].
// Positions p along DIR whose ghost source is i: p = i, plus the ghost images (periodic
// wrap, lower mirror -1-i, upper shifted copy i+3) that lie in the stencil range [-3, n+2].
template <int NCHEM, int DIR>
__global__ void __launch_bounds__(256) vjp_gather_kernel(Grid g, const double* __restrict__ A,
                                                         Fields u, long nfaces, int first) {
  constexpr int NV = 5 + NCHEM;
  const long nx = g.n[0], ny = g.n[1], nd = g.n[DIR];
  const int blo = g.bc[2 * DIR], bhi = g.bc[2 * DIR + 1];
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < g.ncell;
       c += (long)gridDim.x * blockDim.x) {
    long i0, j0, k0;
    split3(c, nx, ny, i0, j0, k0);
    const long pos[3] = {i0, j0, k0};
    const long id = pos[DIR];
    long cand[4];
    int nc = 0;
    cand[nc++] = id;
    if (blo == GBMV_BC_PERIODIC) {
      if (id - nd >= -3) cand[nc++] = id - nd;
      if (id + nd <= nd + 2) cand[nc++] = id + nd;
    } else {
      if (-1 - id >= -3) cand[nc++] = -1 - id;
      if (id + 3 >= nd && id + 3 <= nd + 2) cand[nc++] = id + 3;
    }
    (void)bhi;
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    for (int q = 0; q < nc; ++q) {
      const long p = cand[q];
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        const long fd = p + 3 - l;  // face index along DIR whose slot l sits at p
        if (fd < 0 || fd > nd) continue;
        long fp[3] = {pos[0], pos[1], pos[2]};
        fp[DIR] = fd;
        const long ex = nx + (DIR == 0), ey = ny + (DIR == 1);
        const long f = fp[0] + ex * (fp[1] + ey * fp[2]);
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] += A[((long)l * NV + v) * nfaces + f];
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double* dst = (v < 5) ? (u.f[v] + c) : (u.f[5] + (v - 5) + (long)NCHEM * c);
      *dst = first ? acc[v] : *dst + acc[v];
    }
  }
}

// ------------------------------------------------------------------ launcher

template <int NCHEM, int DIR>
static int vjp_dir(const Grid& g, const SweepSet& S, const Fields& out, double* A,
                   cudaStream_t s) {
  const long nf = S.d[DIR].nfaces;
  const int t = spread_threads(nf, 128);
  face_flux_vjp_kernel<NCHEM><<<sweep_blocks(nf, t), t, 0, s>>>(S, DIR, g.inv_d[DIR], A);
  GBMV_LAUNCH_CHECK("face_flux_vjp_kernel");
  vjp_gather_kernel<NCHEM, DIR><<<sweep_blocks(g.ncell, 256), 256, 0, s>>>(g, A, out, nf, DIR == 0);
  GBMV_LAUNCH_CHECK("vjp_gather_kernel");
  return GBMV_OK;
}

template <int NCHEM>
static int vjp_t(const Grid& g, const Fields& w, const Fields& v, const Fields& out, double* A,
                 cudaStream_t s) {
  ProfScope ps("vjp", s);
  // cell primitives after the stencil cotangents (not in the flux scratch: a flux divergence on
  // the same handle may run beside the adjoint on another stream)
  double* const q = A + feuler_vjp_scratch_doubles(g) - 5 * g.ncell;
  double* const p[5] = {q, q + g.ncell, q + 2 * g.ncell, q + 3 * g.ncell, q + 4 * g.ncell};
  int rc = prims64(g, w, p, nullptr, s);
  SweepSet S;
  sweep_set(g, w, nullptr, 1, 128, (long)kSM * 16, S);
  sweep_second(S, v);
  const double* const u[3] = {p[1], p[2], p[3]};
  sweep_prims(S, p[0], u, p[4]);
  if (!rc) rc = vjp_dir<NCHEM, 0>(g, S, out, A, s);
  if (!rc) rc = vjp_dir<NCHEM, 1>(g, S, out, A, s);
  if (!rc) rc = vjp_dir<NCHEM, 2>(g, S, out, A, s);
  return rc;
}

size_t feuler_vjp_scratch_doubles(const Grid& g) {
  const long nx = g.n[0], ny = g.n[1], nz = g.n[2];
  long m = (nx + 1) * ny * nz;
  if (nx * (ny + 1) * nz > m) m = nx * (ny + 1) * nz;
  if (nx * ny * (nz + 1) > m) m = nx * ny * (nz + 1);
  return (size_t)6 * (5 + g.nchem) * (size_t)m + 5 * (size_t)g.ncell;
}

int feuler_vjp(const Grid& g, const Fields& w, const Fields& v, const Fields& out, double* A,
               cudaStream_t s) {
  switch (g.nchem) {
    case 0: return vjp_t<0>(g, w, v, out, A, s);
    case 2: return vjp_t<2>(g, w, v, out, A, s);
    case 4: return vjp_t<4>(g, w, v, out, A, s);
    case 6: return vjp_t<6>(g, w, v, out, A, s);
    case 10: return vjp_t<10>(g, w, v, out, A, s);
    default: return GBMV_EUNSUPPORTED;
  }
}

}  // namespace gbmv
