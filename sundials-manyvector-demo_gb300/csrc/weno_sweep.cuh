// Face indexing and stencil gather shared by every face-sweep kernel (the FP64 and float-float
// face fluxes, pack1D, the JVP and VJP sweeps).
//
// A sweep normal to DIR visits every face of the (n_DIR + 1) per row, the lower faces of all
// cells plus the upper boundary faces, as the reference's interior and boundary flux loops do
// together (src/utilities.cpp:17-253).  Face f has coordinates (i, j, k) in the face grid of
// extents n + e_DIR; its stencil points sit at positions i_DIR - 3 .. i_DIR + 2 along DIR and
// take their values through the ghost rule of common.cuh (ghost_src).
#pragma once

#include "common.cuh"
#include "weno.cuh"

namespace gbmv {

// (i, j, k) of the linear index c = i + ex (j + ey k): 32-bit unsigned division while c fits
// (a 64-bit division is a long emulated sequence, comparable to the rest of a cheap pass)
__device__ __forceinline__ void split3(long c, long ex, long ey, long& i, long& j, long& k) {
  if ((unsigned long)c <= 0xffffffffUL) {
    const unsigned u = (unsigned)c, ux = (unsigned)ex, uy = (unsigned)ey;
    const unsigned r = u / ux, q = r / uy;
    i = (long)(u - r * ux);
    j = (long)(r - q * uy);
    k = (long)q;
  } else {
    const long r = c / ex, q = r / ey;
    i = c - r * ex;
    j = r - q * ey;
    k = q;
  }
}

template <int DIR>
__device__ __forceinline__ void face_coords(long f, const Grid& g, long& i, long& j, long& k) {
  split3(f, g.n[0] + (DIR == 0), g.n[1] + (DIR == 1), i, j, k);
}

// One direction of a sweep that takes the direction at run time: one kernel body serves the
// three, and one launch covers the faces of all of them (SweepSet), so small grids wait for one
// sweep instead of three in a row.  Field order as load_point: normal momentum in slot 1.
struct SweepDir {
  const double* f[5];  // rho, m_normal, m_t1, m_t2, et
  int slot[5];         // their field numbers
  const double* g[5];  // a second ManyVector in the same order (tangents; null: none)
  const double* vel[3];  // velocities: normal, t1, t2 (null: no primitives)
  double* F;           // face fluxes [field][face]
  long nfaces, ex, ey; // extents of the face grid along x and y
  long n, stride;      // cells along the direction and their spacing in memory
  int dir, bc_lo, bc_hi;
  int block0;          // first block of the direction
};
struct SweepSet {
  SweepDir d[3];
  const double* ph;    // half pressure, half sound speed (null: no primitives)
  const double* hc;
  const double* chem;
  const double* gchem; // the second ManyVector's tracers
  long nx, ny;
  double gamma;
};
__device__ __forceinline__ int sweep_dir(const SweepSet& S) {
  return (int)blockIdx.x >= S.d[2].block0 ? 2 : ((int)blockIdx.x >= S.d[1].block0 ? 1 : 0);
}

// cells and ghost signs of the six stencil points of face f of a direction, point l at stencil
// position l, or 5 - l when reversed
__device__ __forceinline__ void stencil_of(const SweepSet& S, const SweepDir& D, long f,
                                           bool reversed, long (&cell)[6], bool (&nall)[6],
                                           bool (&nnorm)[6]) {
  long i, j, k;
  split3(f, D.ex, D.ey, i, j, k);
  const long pos = D.dir == 0 ? i : (D.dir == 1 ? j : k);
  const long base = i + S.nx * (j + S.ny * k) - pos * D.stride;
#pragma unroll
  for (int l = 0; l < 6; ++l)
    cell[l] = base + D.stride * ghost_src(pos - 3 + (reversed ? 5 - l : l), D.n, D.bc_lo, D.bc_hi,
                                          &nall[l], &nnorm[l]);
}

// the fluid values of a stencil point in face order, ghost signs applied
__device__ __forceinline__ void load_point(const double* const (&f)[5], long c, bool nall,
                                           bool nnorm, double (&W)[5]) {
#pragma unroll
  for (int v = 0; v < 5; ++v) W[v] = flip_sign(__ldg(f[v] + c), nall != (v == 1 && nnorm));
}

// grid-stride launch size: ceil(n / t) blocks, at least 1, at most 16 per SM
inline int sweep_blocks(long n, int t) {
  long b = (n + t - 1) / t;
  const long cap = (long)kSM * 16;
  return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

// Threads per block of a one-item-per-thread pass over n items whose kernel allows up to
// tmax: the largest of tmax, tmax/2, ..., 32 that still gives every SM two blocks, so that a
// small grid (the Sod tube's ~1200 faces) spreads over as many SMs as it can fill instead of
// queueing its FP64 work on a few of them; large grids keep tmax.  Each item is computed by
// one thread independently, so the results do not depend on the choice.
inline int spread_threads(long n, int tmax) {
  int t = tmax;
  while (t > 32 && n < 2L * kSM * t) t /= 2;
  return t;
}

// the face sweeps' threads per block: the tuned value, else by size
inline int sweep_threads(const Grid& g, long n, int tmax) {
  return g.sweep_threads > 0 && g.sweep_threads <= tmax ? g.sweep_threads
                                                        : spread_threads(n, tmax);
}

// faces normal to x, y, z
inline void face_counts(const Grid& g, long (&nf)[3]) {
  const long nx = g.n[0], ny = g.n[1], nz = g.n[2];
  nf[0] = (nx + 1) * ny * nz;
  nf[1] = nx * (ny + 1) * nz;
  nf[2] = nx * ny * (nz + 1);
}

// the cell primitives (half pressure, three velocities, half sound speed) of a sweep
inline void sweep_prims(SweepSet& S, const double* ph, const double* const (&u)[3],
                        const double* hc) {
  S.ph = ph;
  S.hc = hc;
  for (int d = 0; d < 3; ++d) {
    S.d[d].vel[0] = u[d];
    S.d[d].vel[1] = u[d == 0 ? 1 : (d == 1 ? 0 : 1)];
    S.d[d].vel[2] = u[d == 2 ? 0 : 2];
  }
}

// a second ManyVector read beside w
inline void sweep_second(SweepSet& S, const Fields& v) {
  for (int d = 0; d < 3; ++d)
    for (int k = 0; k < 5; ++k) S.d[d].g[k] = v.f[S.d[d].slot[k]];
  S.gchem = v.f[5];
}

// The three directions of w for a sweep of `per_face` threads a face in blocks of t threads,
// fluxes to F (null: none); returns the number of blocks (at most cap per direction).
inline int sweep_set(const Grid& g, const Fields& w, double* const* F, int per_face, int t,
                     long cap, SweepSet& S) {
  long nf[3], b = 0;
  face_counts(g, nf);
  const long stride[3] = {1, g.n[0], g.n[0] * g.n[1]};
  for (int d = 0; d < 3; ++d) {
    SweepDir& D = S.d[d];
    const int slot[5] = {0, 1 + d, d == 1 ? 1 : 2, d == 2 ? 1 : 3, 4};
    for (int v = 0; v < 5; ++v) {
      D.slot[v] = slot[v];
      D.f[v] = w.f[slot[v]];
    }
    for (int v = 0; v < 5; ++v) D.g[v] = nullptr;
    for (int v = 0; v < 3; ++v) D.vel[v] = nullptr;
    D.F = F ? F[d] : nullptr;
    D.nfaces = nf[d];
    D.ex = g.n[0] + (d == 0);
    D.ey = g.n[1] + (d == 1);
    D.n = g.n[d];
    D.stride = stride[d];
    D.dir = d;
    D.bc_lo = g.bc[2 * d];
    D.bc_hi = g.bc[2 * d + 1];
    D.block0 = (int)b;
    const long nb = (nf[d] * per_face + t - 1) / t;
    b += nb < cap ? nb : cap;
  }
  S.ph = S.hc = nullptr;
  S.chem = w.f[5];
  S.gchem = nullptr;
  S.nx = g.n[0];
  S.ny = g.n[1];
  S.gamma = g.gamma;
  return (int)b;
}

}  // namespace gbmv
