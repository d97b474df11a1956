// Float-float (mixed) form of the WENO flux divergence (src/utilities.cpp:17-253):
//
//   prims_f2_kernel: once per cell, in FP64 exactly as the reference evaluates them per
//     stencil point -- pressure (eos), the three velocities m/rho and the sound speed
//     sqrt(gamma p / rho) -- then every field and primitive split into float pairs (hi, lo):
//     Q2[q][cell], q = rho, mx, my, mz, et, p, ux, uy, uz, c, tracers...;
//   fluid_flux_f2_kernel: the five fluid face fluxes of the three directions in float-float
//     arithmetic from Q2 (no FP64 instruction on the common path), the two Lax-Friedrichs sides of
//     every reconstruction evaluated together on the paired FP32 instructions (df64x2.cuh);
//     faces whose states leave the float range, or touch a non-positive density (homogeneous
//     Dirichlet ghosts), are computed in FP64 from w;
//   tracer_flux_f2_kernel<WV>: the tracers' face fluxes, WV = 0 with float-float weights, WV = 1
//     with FP32 weights and smoothness indicators in correction form;
//   divergence_f2: the FP64 form's divergence pass over fluxes kept as float pairs, the
//     differences in float-float, the final G - div in FP64 (weno.cu).
//
// Fluid and tracers are separate launches because their registers are: the fluid part holds a
// stencil, its projections and the eigenvectors (168 registers under the alone budget, 10-12
// warps per SM), a tracer only its split factors, and the sweep is bound by FP32 latency, so the
// tracers run at two to three times the warps.
#pragma once

#include "common.cuh"
#include "weno_face.cuh"
#include "weno_sweep.cuh"

namespace gbmv {

constexpr int kQ2Base = 10;  // index of the first tracer in Q2

// Q2 from w, and the legal-state flags OR-ed into *d_status (weno_f2.cu)
int prims_f2(const Grid& g, const Fields& w, float2* q2, const double* tscale, int* d_status,
             cudaStream_t s);

// float-float primitive q of stencil cell c
__device__ __forceinline__ f2 q2_load(const float2* __restrict__ Q2, long n, int q, unsigned c) {
  const float2 t = __ldg(Q2 + (long)q * n + c);
  return f2(t.x, t.y);
}

// The stencil of a face: cells and, as bit masks over its points, the ghost signs.
struct StencilF2 {
  unsigned cell[6];
  unsigned nall, nnorm;
};
__device__ __forceinline__ void stencil_f2(const SweepSet& S, const SweepDir& D, long f,
                                           StencilF2& T) {
  long cell[6];
  bool nall[6], nnorm[6];
  stencil_of(S, D, f, false, cell, nall, nnorm);
  T.nall = T.nnorm = 0;
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    T.cell[l] = (unsigned)cell[l];  // (cell counts are far below 2^32: ~280 bytes per cell)
    T.nall |= (unsigned)nall[l] << l;
    T.nnorm |= (unsigned)nnorm[l] << l;
  }
}

}  // namespace gbmv
