// WENO5 flux divergence (part a): the device implementation of fEuler
// (src/utilities.cpp:17-253) with in-kernel ghost synthesis for every boundary type.
//
// FP64 parity form, three passes:
//   1. prims64_kernel: the primitives of every cell into the tendency arrays (which the last pass
//      overwrites), and the legal-state check (src/euler3D.hpp:1405-1414) OR-ed into a status
//      word.
//   2. face_flux64_kernel<NCHEM, PRE, SPLIT>: the faces of the three directions in one launch, a
//      thread a face (all lower faces plus the upper boundary faces, like the reference's two
//      loops), two or four threads on small grids; stencil gathered straight from the SoA fields
//      with ghost synthesis, flux written to a per-direction scratch array F_DIR[v][face] (the
//      xflux/yflux/zflux arrays of EulerData, src/euler3D.hpp:497-499, stored field-major so that
//      the divergence pass reads them coalesced).
//   3. divergence_kernel<NCHEM>: wdot = G - [(Fx+ - Fx-)/dx + (Fy+ - Fy-)/dy + (Fz+ - Fz-)/dz].
// The float-float forms (weno_f2.cu) use divergence_f2_kernel below as their last pass.  Also
// here: the CFL wave speed, the pack1D stencil gather, the conservation totals and norms.
#include "common.cuh"
#include "weno64.cuh"
#include "df64.cuh"
#include "weno_sweep.cuh"
#include "weno.cuh"

namespace gbmv {

// Primitives of every cell -- half the pressure, the velocities, half the sound speed -- and the
// legal-state flags (src/euler3D.hpp:1405-1414).  A cell is read by 18 stencil positions, and
// forming its primitives there cost ~45 of a face's FP64 instructions six times over.
__global__ void __launch_bounds__(256) prims64_kernel(Grid g, Fields w, double* ph, double* ux,
                                                      double* uy, double* uz, double* hc,
                                                      int* __restrict__ status) {
  int bad = 0;
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < g.ncell;
       c += (long)gridDim.x * blockDim.x) {
    const double rho = w.f[0][c], mx = w.f[1][c], my = w.f[2][c], mz = w.f[3][c], et = w.f[4][c];
    double p, a;
    point_prims64(g.gamma, rho, mx, my, mz, et, p, a);
    bad |= (!(rho > 0.0) ? 1 : 0) | (!(et > 0.0) ? 2 : 0) | (!(p > 0.0) ? 4 : 0);
    if (ph) {
      ph[c] = p;
      ux[c] = mx / rho;
      uy[c] = my / rho;
      uz[c] = mz / rho;
      hc[c] = a;
    }
  }
  bad = __reduce_or_sync(0xffffffffu, bad);
  if (status && bad && (threadIdx.x & 31) == 0) atomicOr(status, bad);
}

int prims64(const Grid& g, const Fields& w, double* const (&out)[5], int* d_status,
            cudaStream_t s) {
  ProfScope ps("prims", s);
  const int t = spread_threads(g.ncell, 256);
  prims64_kernel<<<sweep_blocks(g.ncell, t), t, 0, s>>>(g, w, out[0], out[1], out[2], out[3],
                                                        out[4], d_status);
  GBMV_LAUNCH_CHECK("prims64_kernel");
  return GBMV_OK;
}

// Face fluxes of the three directions (one launch).  Bound by the FP64 pipe: 1355 instructions
// a face at NVAR 15.  PRE: the primitives are read from the cell pass, else formed per stencil
// point.  SPLIT: two neighbouring threads share a face, each with one Lax-Friedrichs side (the
// second reads its stencil reversed, which makes its side the plus formula); the same bits.
template <int NCHEM, bool PRE, bool SPLIT>
__global__ void __launch_bounds__(128) face_flux64_kernel(const __grid_constant__ SweepSet S) {
  const int dir = sweep_dir(S);
  const SweepDir& D = S.d[dir];
  const int nblk = (dir == 2 ? (int)gridDim.x : S.d[dir + 1].block0) - D.block0;
  const long first = (blockIdx.x - D.block0) * (long)blockDim.x + threadIdx.x;
  const int side = SPLIT ? (int)(threadIdx.x & 1) : 0;
  // SPLIT: one pass (the launch covers every face); surplus threads repeat the last face so that
  // both threads of a pair and the whole warp reach the exchanges
  for (long f = SPLIT ? (first >> 1) : first; SPLIT || f < D.nfaces;
       f += (long)nblk * blockDim.x) {
    const bool live = f < D.nfaces;
    if (SPLIT && !live) f = D.nfaces - 1;
    long cell[6];
    bool nall[6], nnorm[6];
    stencil_of(S, D, f, side, cell, nall, nnorm);
    Stencil64 T;
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      load_point(D.f, cell[l], nall[l], nnorm[l], T.W[l]);
      if (PRE) {
        const double p = __ldg(S.ph + cell[l]), u = __ldg(D.vel[0] + cell[l]);
        T.ph[l] = flip_sign(p, nall[l]);
        T.u[l] = flip_sign(u, nnorm[l]);
        T.hc[l] = __ldg(S.hc + cell[l]);
      } else {
        point_prims64(S.gamma, T.W[l][0], T.W[l][1], T.W[l][2], T.W[l][3], T.W[l][4], T.ph[l],
                      T.hc[l]);
        T.u[l] = T.W[l][1] / T.W[l][0];
      }
    }
    if constexpr (!SPLIT) {
      Split64 H;
      double out[5];
      fluid_face_flux64<(NCHEM > 0)>(T, S.gamma, H, out);
#pragma unroll
      for (int v = 0; v < 5; ++v) D.F[D.slot[v] * D.nfaces + f] = out[v];
#pragma unroll 1
      for (int c = 0; c < NCHEM; ++c) {
        double cv[6];
#pragma unroll
        for (int l = 0; l < 6; ++l) {
          cv[l] = flip_sign(__ldg(S.chem + c + (long)NCHEM * cell[l]), nall[l]);
        }
        D.F[(5 + c) * D.nfaces + f] = tracer_face_flux64(H, cv);
      }
    } else {
      Roe64 R;
      roe64(T, S.gamma, R);
      const double ha = half_alpha64(T);
      double h[5], ff[5], out[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) h[k] = fma(0.5, T.u[k], side ? -ha : ha);
      fluid_side64<0>(T, R, h, ff);
#pragma unroll
      for (int i = 0; i < 5; ++i) ff[i] += __shfl_xor_sync(0xffffffffu, ff[i], 1);
      fluid_back64(R, ff, out);
#pragma unroll
      for (int v = 0; v < 5; ++v)
        if (live && (v & 1) == side) D.F[D.slot[v] * D.nfaces + f] = out[v];
#pragma unroll 1
      for (int c = 0; c < NCHEM; ++c) {
        double cv[5];
#pragma unroll
        for (int l = 0; l < 5; ++l) {
          cv[l] = flip_sign(__ldg(S.chem + c + (long)NCHEM * cell[l]), nall[l]);
        }
        Weno64 q;
        double r =
            weno_prod64<true>(cv[0], h[0], cv[1], h[1], cv[2], h[2], cv[3], h[3], cv[4], h[4], q);
        r += __shfl_xor_sync(0xffffffffu, r, 1);
        if (live && (c & 1) == side) D.F[(5 + c) * D.nfaces + f] = r;
      }
      break;
    }
  }
}

// The same for the smallest grids, four threads a face: a lane pair per face as above in each of
// the block's two warps, which share the characteristic components (66 and 99 of the 165 FP64
// instructions of a side's reconstructions) and the tracers.  The device
// time of a right-hand side, two threads a face and four: 128 x 3 x 3 without tracers 26.7 and 24.6
// us, 10^3 with ten 47.1 and 36.9 (a warp issues its FP64 chain at one instruction per 64 cycles
// whatever its lanes hold, so only further warps shorten it).  The same bits.
template <int NCHEM>
__global__ void __launch_bounds__(64) face_flux64_quad_kernel(const __grid_constant__ SweepSet S) {
  __shared__ double share[5][16];
  const int dir = sweep_dir(S);
  const SweepDir& D = S.d[dir];
  const int side = threadIdx.x & 1, half = threadIdx.x >> 5, slot = (threadIdx.x & 31) >> 1;
  long f = (blockIdx.x - D.block0) * 16L + slot;
  const bool live = f < D.nfaces;
  if (!live) f = D.nfaces - 1;  // surplus threads repeat the last face and store nothing
  long cell[6];
  bool nall[6], nnorm[6];
  stencil_of(S, D, f, side, cell, nall, nnorm);
  Stencil64 T;
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    load_point(D.f, cell[l], nall[l], nnorm[l], T.W[l]);
    T.ph[l] = flip_sign(__ldg(S.ph + cell[l]), nall[l]);
    T.u[l] = flip_sign(__ldg(D.vel[0] + cell[l]), nnorm[l]);
    T.hc[l] = __ldg(S.hc + cell[l]);
  }
  Roe64 R;
  roe64(T, S.gamma, R);
  const double ha = half_alpha64(T);
  double h[5], ff[5] = {0, 0, 0, 0, 0}, out[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) h[k] = fma(0.5, T.u[k], side ? -ha : ha);
  if (half) fluid_side64<0, 2>(T, R, h, ff);
  else fluid_side64<0, 1>(T, R, h, ff);
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const double o = __shfl_xor_sync(0xffffffffu, ff[i], 1);
    if ((half == 0) == (i == 0 || i == 4) && side == 0) share[i][slot] = ff[i] + o;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 5; ++i) ff[i] = share[i][slot];
  fluid_back64(R, ff, out);
#pragma unroll
  for (int v = 0; v < 5; ++v)
    if (live && (v & 3) == 2 * half + side) D.F[D.slot[v] * D.nfaces + f] = out[v];
#pragma unroll 1
  for (int c = half; c < NCHEM; c += 2) {
    double cv[5];
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      cv[l] = flip_sign(__ldg(S.chem + c + (long)NCHEM * cell[l]), nall[l]);
    }
    Weno64 q;
    double r =
        weno_prod64<true>(cv[0], h[0], cv[1], h[1], cv[2], h[2], cv[3], h[3], cv[4], h[4], q);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    if (live && side == 0) D.F[(5 + c) * D.nfaces + f] = r;
  }
}

template <int NCHEM>
__global__ void __launch_bounds__(256) divergence_kernel(Grid g, Fields wdot,
                                                         const double* __restrict__ Fx,
                                                         const double* __restrict__ Fy,
                                                         const double* __restrict__ Fz,
                                                         ForceTerm G) {
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
      // (F+ - F-) / d as a multiply by 1/d: the reference divides; the difference is one
      // rounding, and 45 FP64 divisions per cell would cost more than the rest of this pass.
      // Subtracted from G as it goes: six FP64 instructions a field
      double* dst = (v < 5) ? (wdot.f[v] + c) : (wdot.f[5] + (v - 5) + (long)NCHEM * c);
      double r = G.in_wdot ? *dst : G.c[v];
      r = fma(Fx[v * nfx + fx] - Fx[v * nfx + fx + 1], g.inv_d[0], r);
      r = fma(Fy[v * nfy + fy] - Fy[v * nfy + fy + nx], g.inv_d[1], r);
      *dst = fma(Fz[v * nfz + fz] - Fz[v * nfz + fz + nx * ny], g.inv_d[2], r);
    }
  }
}

int divergence(const Grid& g, const Fields& wdot, double* const (&F)[3], const ForceTerm& G,
               cudaStream_t s) {
  ProfScope ps("divergence", s);
  const int t = spread_threads(g.ncell, 256);
  const int b = sweep_blocks(g.ncell, t);
  switch (g.nchem) {
    case 0: divergence_kernel<0><<<b, t, 0, s>>>(g, wdot, F[0], F[1], F[2], G); break;
    case 2: divergence_kernel<2><<<b, t, 0, s>>>(g, wdot, F[0], F[1], F[2], G); break;
    case 4: divergence_kernel<4><<<b, t, 0, s>>>(g, wdot, F[0], F[1], F[2], G); break;
    case 6: divergence_kernel<6><<<b, t, 0, s>>>(g, wdot, F[0], F[1], F[2], G); break;
    case 10: divergence_kernel<10><<<b, t, 0, s>>>(g, wdot, F[0], F[1], F[2], G); break;
    default: set_error("nchem=%d not compiled (0,2,4,6,10)", g.nchem); return GBMV_EUNSUPPORTED;
  }
  GBMV_LAUNCH_CHECK("divergence_kernel");
  return GBMV_OK;
}

// Pass 2 of the float-float form: the same divergence over fluxes kept as float pairs.  On
// GB300 the FP64 pipe runs at 1/64 of the FP32 rate, so the divergence's FP64 differences made
// it FP64-bound (81 % of the pipe) at three times its HBM time; here the differences and the
// 1/d scaling are float-float (FP32 pipes) and only G - div is FP64.  The legal-state flags of
// the float-float forms are set by the primitives pass, which already has the pressure, so this
// pass reads no state field and needs no division.
template <int NCHEM>
__global__ void __launch_bounds__(256, 4) divergence_f2_kernel(Grid g, Fields wdot,
                                                            const float2* __restrict__ Fx,
                                                            const float2* __restrict__ Fy,
                                                            const float2* __restrict__ Fz,
                                                            ForceTerm G) {
  const long nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const long nfx = (nx + 1) * ny * nz, nfy = nx * (ny + 1) * nz, nfz = nx * ny * (nz + 1);
  const f2 idx = f2_from_double(g.inv_d[0]), idy = f2_from_double(g.inv_d[1]),
           idz = f2_from_double(g.inv_d[2]);
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < g.ncell;
       c += (long)gridDim.x * blockDim.x) {
    long i, j, k;
    split3(c, nx, ny, i, j, k);
    const long fx = i + (nx + 1) * (j + ny * k);
    const long fy = i + nx * (j + (ny + 1) * k);
    const long fz = c;
    // fields in groups whose 6 fluxes each are loaded before any is used: the rare conversions'
    // branches keep the compiler from moving loads up across them.  128^3 x 15: groups of 2 at 4
    // blocks per SM 234 us; 3 at 3 257; 1 at 6 292; 5 at 3 295, unbounded 381 (290 before)
    constexpr int NV = 5 + NCHEM, GR = 2;
#pragma unroll
    for (int v0 = 0; v0 < NV; v0 += GR) {
      float2 x[GR][6];
#pragma unroll
      for (int q = 0; q < GR; ++q) {
        const int v = v0 + q;
        if (v < NV) {
          x[q][0] = Fx[v * nfx + fx + 1];
          x[q][1] = Fx[v * nfx + fx];
          x[q][2] = Fy[v * nfy + fy + nx];
          x[q][3] = Fy[v * nfy + fy];
          x[q][4] = Fz[v * nfz + fz + nx * ny];
          x[q][5] = Fz[v * nfz + fz];
        }
      }
#pragma unroll
      for (int q = 0; q < GR; ++q) {
        const int v = v0 + q;
        if (v < NV) {
          const f2 div = (f2(x[q][0].x, x[q][0].y) - f2(x[q][1].x, x[q][1].y)) * idx +
                         (f2(x[q][2].x, x[q][2].y) - f2(x[q][3].x, x[q][3].y)) * idy +
                         (f2(x[q][4].x, x[q][4].y) - f2(x[q][5].x, x[q][5].y)) * idz;
          double* dst = (v < 5) ? (wdot.f[v] + c) : (wdot.f[5] + (v - 5) + (long)NCHEM * c);
          const double base = G.in_wdot ? *dst : G.c[v];
          *dst = base - f2_to_double(div);
        }
      }
    }
  }
}

int divergence_f2(const Grid& g, const Fields& wdot, float2* const (&F)[3], const ForceTerm& G,
                  cudaStream_t s) {
  ProfScope ps("divergence", s);
  const int b = sweep_blocks(g.ncell, 256);
  switch (g.nchem) {
#define GBMV_DIV_F2(NC)                                                     \
  case NC:                                                                  \
    divergence_f2_kernel<NC><<<b, 256, 0, s>>>(g, wdot, F[0], F[1], F[2], G); \
    break;
    GBMV_DIV_F2(0)
    GBMV_DIV_F2(2)
    GBMV_DIV_F2(4)
    GBMV_DIV_F2(6)
    GBMV_DIV_F2(10)
#undef GBMV_DIV_F2
    default: set_error("nchem=%d not compiled (0,2,4,6,10)", g.nchem); return GBMV_EUNSUPPORTED;
  }
  GBMV_LAUNCH_CHECK("divergence_f2_kernel");
  return GBMV_OK;
}

// Whether w and the five fluid tendencies share memory (an in-place call)
bool fields_overlap(const Grid& g, const Fields& w, const Fields& wdot) {
  for (int a = 0; a < 5; ++a)
    for (int b = 0; b < (g.nchem ? 6 : 5); ++b) {
      const uintptr_t x = (uintptr_t)wdot.f[a], y = (uintptr_t)w.f[b];
      const uintptr_t nx = 8 * (uintptr_t)g.ncell, ny = nx * (b == 5 ? g.nchem : 1);
      if (x < y + ny && y < x + nx) return true;
    }
  return false;
}

template <int NCHEM>
static int launch_fp64(const Grid& g, const Fields& w, const Fields& wdot, const ForceTerm& G,
                       double* scratch, int* d_status, cudaStream_t s) {
  long nf[3];
  face_counts(g, nf);
  const long nfaces = nf[0] + nf[1] + nf[2];
  double* F[3] = {scratch, scratch + (long)(5 + NCHEM) * nf[0],
                  scratch + (long)(5 + NCHEM) * (nf[0] + nf[1])};
  // The primitives live in the five fluid tendencies, which the divergence overwrites last: no
  // memory of their own.  Where those hold the caller's forcing, or are the state itself, the
  // sweep forms the primitives per stencil point instead.
  const bool pre = !G.in_wdot && !fields_overlap(g, w, wdot);
  {
    double* const none[5] = {};
    double* const out[5] = {wdot.f[0], wdot.f[1], wdot.f[2], wdot.f[3], wdot.f[4]};
    const int rc = prims64(g, w, pre ? out : none, d_status, s);
    if (rc) return rc;
  }
  {
    ProfScope ps("face_flux", s);
    const bool split = pre && nfaces <= kSplitFaces;
    const bool quad = split && nfaces <= kQuadFaces;
    const int per_face = quad ? 4 : (split ? 2 : 1);
    const int t = quad ? 64 : sweep_threads(g, per_face * nfaces, 128);
    SweepSet S;
    const int b = sweep_set(g, w, F, per_face, t, split ? 1L << 30 : (long)kSM * 16, S);
    if (pre) {
      const double* const u[3] = {wdot.f[1], wdot.f[2], wdot.f[3]};
      sweep_prims(S, wdot.f[0], u, wdot.f[4]);
    }
    if (quad) face_flux64_quad_kernel<NCHEM><<<b, t, 0, s>>>(S);
    else if (split) face_flux64_kernel<NCHEM, true, true><<<b, t, 0, s>>>(S);
    else if (pre) face_flux64_kernel<NCHEM, true, false><<<b, t, 0, s>>>(S);
    else face_flux64_kernel<NCHEM, false, false><<<b, t, 0, s>>>(S);
    GBMV_LAUNCH_CHECK("face_flux64_kernel");
  }
  return divergence(g, wdot, F, G, s);
}

size_t feuler_fp64_scratch_doubles(const Grid& g) {
  long nf[3];
  face_counts(g, nf);
  return (size_t)(5 + g.nchem) * (size_t)(nf[0] + nf[1] + nf[2]);
}

int feuler_fp64(const Grid& g, const Fields& w, const Fields& wdot, const ForceTerm& G,
                double* scratch, int* d_status, cudaStream_t s) {
  switch (g.nchem) {
    case 0: return launch_fp64<0>(g, w, wdot, G, scratch, d_status, s);
    case 2: return launch_fp64<2>(g, w, wdot, G, scratch, d_status, s);
    case 4: return launch_fp64<4>(g, w, wdot, G, scratch, d_status, s);
    case 6: return launch_fp64<6>(g, w, wdot, G, scratch, d_status, s);
    case 10: return launch_fp64<10>(g, w, wdot, G, scratch, d_status, s);
    default: set_error("nchem=%d not compiled (0,2,4,6,10)", g.nchem); return GBMV_EUNSUPPORTED;
  }
}

// ------------------------------------------------------------------ CFL-stable step (stability)
//
// stability (src/utilities.cpp:483-528): alpha = max over cells of |mx/rho| + sqrt(gamma p/rho)
// -- the reference takes |mx/rho| for all three directions -- and
// dt = cfl * min(dx, dy, dz) / alpha.  Non-negative doubles order like their bit patterns, so
// the grid maximum is an atomicMax on the 64-bit integer view; NaN cells are skipped, as the
// reference's std::max(alpha, NaN) keeps alpha.

__global__ void __launch_bounds__(256) wave_speed_max_kernel(Grid g, Fields w,
                                                            unsigned long long* __restrict__ out) {
  double m = 0.0;
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < g.ncell;
       c += (long)gridDim.x * blockDim.x) {
    // bound by the FP64 pipe: one reciprocal serves the three quotients (100^3: 92 -> 56 us)
    const double rho = w.f[0][c], mx = w.f[1][c], my = w.f[2][c], mz = w.f[3][c], et = w.f[4][c];
    const double ir = rcp64(rho);
    const double u = fabs(over64(mx, rho, ir));
    const double p = (g.gamma - 1.0) *
                     (et - over64(0.5 * (mx * mx + my * my + mz * mz), rho, ir));
    const double cs = sqrt0_64(over64(g.gamma * p, rho, ir));
    const double a = fabs(u + cs);
    m = (m < a) ? a : m;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double o = __shfl_xor_sync(0xffffffffu, m, off);
    m = (m < o) ? o : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// pack1D_x/y/z and their _bdry variants (src/euler3D.hpp:1197-1378): for every face normal to
// DIR (all (n+1) per row, as the flux loops), the six-point stencil w1d[l][v] the face flux
// reads, ghost rules applied, fields in the ManyVector order (rho, mx, my, mz, et, species),
// written to out[(l * NVAR + v) * nfaces + f].
template <int DIR>
__global__ void __launch_bounds__(128) pack1d_kernel(Grid g, Fields w, double* __restrict__ out,
                                                     long nfaces) {
  const long nx = g.n[0], ny = g.n[1];
  const int nv = 5 + g.nchem;
  for (long f = blockIdx.x * (long)blockDim.x + threadIdx.x; f < nfaces;
       f += (long)gridDim.x * blockDim.x) {
    long i, j, k;
    face_coords<DIR>(f, g, i, j, k);
    const long base[3] = {i, j, k};
    for (int l = 0; l < 6; ++l) {
      bool nall, nnorm;
      long q[3] = {i, j, k};
      q[DIR] = ghost_src(base[DIR] - 3 + l, g.n[DIR], g.bc[2 * DIR], g.bc[2 * DIR + 1], &nall,
                         &nnorm);
      const long c = q[0] + nx * (q[1] + ny * q[2]);
      for (int v = 0; v < nv; ++v) {
        double x = (v < 5) ? w.f[v][c] : w.f[5][(v - 5) + (long)g.nchem * c];
        if (nall || (nnorm && v == 1 + DIR)) x = -x;
        out[((long)l * nv + v) * nfaces + f] = x;
      }
    }
  }
}

int pack1d(const Grid& g, const Fields& w, int dir, double* out, cudaStream_t s) {
  const long nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const long nf[3] = {(nx + 1) * ny * nz, nx * (ny + 1) * nz, nx * ny * (nz + 1)};
  long b = (nf[dir] + 127) / 128;
  if (b > (long)kSM * 16) b = (long)kSM * 16;
  if (dir == 0) pack1d_kernel<0><<<(int)b, 128, 0, s>>>(g, w, out, nf[0]);
  else if (dir == 1) pack1d_kernel<1><<<(int)b, 128, 0, s>>>(g, w, out, nf[1]);
  else pack1d_kernel<2><<<(int)b, 128, 0, s>>>(g, w, out, nf[2]);
  GBMV_LAUNCH_CHECK("pack1d_kernel");
  return GBMV_OK;
}

// check_conservation (src/io.cpp:503-542): grid totals of rho and et.  Deterministic two-pass
// reduction (fixed grid, per-block partial sums, then one block in a fixed order), FP64 with a
// compensated (two-sum) accumulation per thread.
constexpr int kConsBlocks = 1024;

__device__ __forceinline__ void two_sum_acc(double& s, double& c, double x) {
  const double t = s + x;
  const double bp = t - s;
  c += (s - (t - bp)) + (x - bp);
  s = t;
}

// Compensated sum of the n block partials by one block of 256 threads, in a fixed order (strided
// accumulation, then a tree); thread 0 gets the result.  A single thread walking the 1024
// partials issued its ~7 FP64 instructions each at the pipe's one per 64 cycles: 250 us.
__device__ __forceinline__ double sum_partials(const double* __restrict__ part, int n) {
  __shared__ double ws[8], wc[8];
  double s = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) two_sum_acc(s, c, part[i]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double os = __shfl_down_sync(0xffffffffu, s, off);
    c += __shfl_down_sync(0xffffffffu, c, off);
    two_sum_acc(s, c, os);
  }
  if ((threadIdx.x & 31) == 0) {
    ws[threadIdx.x >> 5] = s;
    wc[threadIdx.x >> 5] = c;
  }
  __syncthreads();
  s = threadIdx.x < 8 ? ws[threadIdx.x] : 0.0;
  c = threadIdx.x < 8 ? wc[threadIdx.x] : 0.0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
      const double os = __shfl_down_sync(0xffffffffu, s, off);
      c += __shfl_down_sync(0xffffffffu, c, off);
      two_sum_acc(s, c, os);
    }
  }
  return s + c;
}

__global__ void __launch_bounds__(256) conservation_partial_kernel(long n, const double* rho,
                                                                   const double* et,
                                                                   double* __restrict__ part) {
  double s0 = 0.0, c0 = 0.0, s1 = 0.0, c1 = 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
    two_sum_acc(s0, c0, rho[i]);
    two_sum_acc(s1, c1, et[i]);
  }
  double a = s0 + c0, b = s1 + c1;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, off);
    b += __shfl_down_sync(0xffffffffu, b, off);
  }
  __shared__ double wa[8], wb[8];
  if ((threadIdx.x & 31) == 0) {
    wa[threadIdx.x >> 5] = a;
    wb[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      ta += wa[k];
      tb += wb[k];
    }
    part[blockIdx.x] = ta;
    part[kConsBlocks + blockIdx.x] = tb;
  }
}

// block 0: rho, block 1: et
__global__ void __launch_bounds__(256) conservation_final_kernel(const double* __restrict__ part,
                                                                 double* __restrict__ out) {
  const double t = sum_partials(part + blockIdx.x * kConsBlocks, kConsBlocks);
  if (threadIdx.x == 0) out[blockIdx.x] = t;
}

int conservation_sums(const Grid& g, const Fields& w, double* d_scratch, double* out,
                      cudaStream_t s) {
  conservation_partial_kernel<<<kConsBlocks, 256, 0, s>>>(g.ncell, w.f[0], w.f[4], d_scratch);
  GBMV_LAUNCH_CHECK("conservation_partial_kernel");
  conservation_final_kernel<<<2, 256, 0, s>>>(d_scratch, out);
  GBMV_LAUNCH_CHECK("conservation_final_kernel");
  return GBMV_OK;
}

// s + x for non-negative numbers, the addition's rounding error added to c: Dekker's sum of the
// larger and the smaller, four FP64 instructions where two_sum_acc takes seven for the same error.
// The order is found on the bits, which for non-negative doubles is integer work (comparisons of
// doubles run on the FP64 pipe).
__device__ __forceinline__ void pos_sum_acc(double& s, double& c, double x) {
  const bool swap = __double_as_longlong(x) > __double_as_longlong(s);
  const double a = swap ? x : s, b = swap ? s : x;
  const double t = a + b;
  c += b - (t - a);
  s = t;
}

// N_VWrmsNorm of the six-component ManyVector (the norm ARKODE's error test and Newton
// convergence test take, src/imex_chem_hydro_main.cpp:463): ewt = 1 / (rtol |y| + atol) per
// entry, sum of (v ewt)^2 over the five fluid fields (ncell each) and the chemistry field
// (nchem ncell), divided by the total length, square root.  Same fixed-grid compensated
// two-pass reduction as the conservation totals, every term compensated; partials in
// scratch[0..kConsBlocks).
__global__ void __launch_bounds__(256) wrms_partial_kernel(long ncell, int nchem, Fields v,
                                                           Fields y, double rtol, double atol,
                                                           double* __restrict__ part) {
  double s0 = 0.0, c0 = 0.0;
  for (int k = 0; k < 6; ++k) {
    const long n = (k < 5) ? ncell : (long)nchem * ncell;
    const double* __restrict__ vk = v.f[k];
    const double* __restrict__ yk = y.f[k];
    if (n == 0) continue;
    // Bound by the FP64 pipe: 11 instructions a term, five of them the weight's reciprocal and
    // four the compensated addition (an IEEE division and two_sum_acc: 18).  100^3 x 15: 408 us
    // with those, 296 now; 228 with one compensation for four terms, which was up to an ulp off.
    // Four terms at a time keep enough loads in flight.
    const long stride = (long)gridDim.x * blockDim.x;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long e = i + j * stride;
        if (e < n) {
          const double q = vk[e] * rcp64_any(fma(rtol, fabs(yk[e]), atol));
          pos_sum_acc(s0, c0, q * q);
        }
      }
    }
  }
  double a = s0 + c0;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) a += __shfl_down_sync(0xffffffffu, a, off);
  __shared__ double wa[8];
  if ((threadIdx.x & 31) == 0) wa[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) ta += wa[k];
    part[blockIdx.x] = ta;
  }
}

__global__ void __launch_bounds__(256) wrms_final_kernel(const double* __restrict__ part,
                                                         double ntotal, double* __restrict__ out) {
  const double t = sum_partials(part, kConsBlocks);
  if (threadIdx.x == 0) out[0] = sqrt(t / ntotal);
}

int wrms_norm(const Grid& g, const Fields& v, const Fields& y, double rtol, double atol,
              double* d_scratch, double* out, cudaStream_t s) {
  wrms_partial_kernel<<<kConsBlocks, 256, 0, s>>>(g.ncell, g.nchem, v, y, rtol, atol, d_scratch);
  GBMV_LAUNCH_CHECK("wrms_partial_kernel");
  const double ntotal = (double)(5 + g.nchem) * (double)g.ncell;
  wrms_final_kernel<<<1, 256, 0, s>>>(d_scratch, ntotal, out);
  GBMV_LAUNCH_CHECK("wrms_final_kernel");
  return GBMV_OK;
}

// print_stats (src/io.cpp:552-640): per field the root mean square over the grid,
// sqrt(sum_cells (x * units)^2 / ncells), fluid fields in code units times the density,
// momentum and energy units (1 for dimensionless output), the chemistry fields as stored.
// Same fixed-grid compensated two-pass reduction as the conservation totals; partials in
// scratch[v * kConsBlocks + block], results in scratch[16 * kConsBlocks + v].
constexpr int kRmsMaxFields = 16;

template <int NCHEM>
__global__ void __launch_bounds__(256) field_rms_partial_kernel(long n, Fields w, double du,
                                                                double mu, double eu,
                                                                double* __restrict__ part) {
  constexpr int NV = 5 + NCHEM;
  double s[NV], c[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) s[v] = c[v] = 0.0;
  const double u[5] = {du, mu, mu, mu, eu};
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double x = w.f[v][i] * u[v];
      two_sum_acc(s[v], c[v], x * x);
    }
#pragma unroll
    for (int v = 0; v < NCHEM; ++v) {
      const double x = w.f[5][v + (long)NCHEM * i];
      two_sum_acc(s[5 + v], c[5 + v], x * x);
    }
  }
  __shared__ double wsum[8][NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double a = s[v] + c[v];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a += __shfl_down_sync(0xffffffffu, a, off);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5][v] = a;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += wsum[k][threadIdx.x];
    part[threadIdx.x * kConsBlocks + blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(256) field_rms_final_kernel(const double* __restrict__ part,
                                                              double ncell,
                                                              double* __restrict__ out) {
  const double t = sum_partials(part + blockIdx.x * kConsBlocks, kConsBlocks);
  if (threadIdx.x == 0) out[blockIdx.x] = sqrt(t / ncell);
}

size_t reduction_scratch_doubles() { return (size_t)kRmsMaxFields * kConsBlocks + kRmsMaxFields; }

int field_rms(const Grid& g, const Fields& w, double du, double mu, double eu, double* d_scratch,
              cudaStream_t s) {
  switch (g.nchem) {
#define GBMV_RMS(NC)                                                                   \
  case NC:                                                                            \
    field_rms_partial_kernel<NC><<<kConsBlocks, 256, 0, s>>>(g.ncell, w, du, mu, eu,   \
                                                            d_scratch);               \
    break;
    GBMV_RMS(0)
    GBMV_RMS(2)
    GBMV_RMS(4)
    GBMV_RMS(6)
    GBMV_RMS(10)
#undef GBMV_RMS
    default: set_error("nchem=%d not compiled (0,2,4,6,10)", g.nchem); return GBMV_EUNSUPPORTED;
  }
  GBMV_LAUNCH_CHECK("field_rms_partial_kernel");
  field_rms_final_kernel<<<5 + g.nchem, 256, 0, s>>>(d_scratch, (double)g.ncell,
                                                     d_scratch + (size_t)kRmsMaxFields * kConsBlocks);
  GBMV_LAUNCH_CHECK("field_rms_final_kernel");
  return GBMV_OK;
}

int wave_speed_max(const Grid& g, const Fields& w, unsigned long long* d_out, cudaStream_t s) {
  long b = (g.ncell + 255) / 256;
  if (b > (long)kSM * 8) b = (long)kSM * 8;
  if (b < 1) b = 1;
  GBMV_CUDA_TRY(cudaMemsetAsync(d_out, 0, sizeof(unsigned long long), s));
  wave_speed_max_kernel<<<(int)b, 256, 0, s>>>(g, w, d_out);
  GBMV_LAUNCH_CHECK("wave_speed_max_kernel");
  return GBMV_OK;
}

}  // namespace gbmv

