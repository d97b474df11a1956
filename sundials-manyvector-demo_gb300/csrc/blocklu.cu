// Block-diagonal Newton linear solve (part c): batched LU with partial pivoting of the 10x10
// chemistry blocks (what SUNLinSol_MagmaDense does with MAGMA's batched getrf/getrs under the
// reference's SUNLinSol_RankLocalLS / SUNLinSol_BDMPIMV wrappers,
// src/multirate_chem_hydro_main.cpp:1312-1411, src/imex_chem_hydro_main.cpp:1075-1194).
//
// One thread owns one block; the whole 10x10 block lives in registers (fully unrolled through
// template recursion, compile-time indices), row interchanges are predicated selects.  A CTA is
// one warp with a tile of 32 consecutive blocks (25.6 KB, contiguous in HBM) brought into shared
// memory by 16-byte asynchronous copies, all in flight at once; several such CTAs per SM overlap
// one tile's traffic with the others' arithmetic.  (Two-warp CTAs filling their tile with plain
// loads, a few in flight, left the FP64 pipe 54 % busy in the factorisation and 20 % in the
// solve: 192,000 blocks 286 and 164 us, now 165 and 59.)
#include "block_tile.cuh"
#include "chem.cuh"
#include "chem_lu.cuh"
#include "weno64.cuh"

namespace gbmv {

// Solve with the factor of lu10_regs in shared memory (row interchanges, unit-lower forward
// substitution, upper back substitution multiplying by the stored reciprocal pivots); columns
// are read in 16-byte pairs, without bank conflicts at this stride.
__device__ __forceinline__ void lus10(const double* __restrict__ A, const int (&piv)[10],
                                      double (&x)[10]) {
#pragma unroll
  for (int kk = 0; kk < 10; ++kk) {
#pragma unroll
    for (int r = kk + 1; r < 10; ++r) {
      const bool sw = (r == piv[kk]);
      const double a = x[kk], b = x[r];
      x[kk] = sw ? b : a;
      x[r] = sw ? a : b;
    }
  }
  const double2* const C = reinterpret_cast<const double2*>(A);
#pragma unroll
  for (int col = 0; col < 9; ++col) {
#pragma unroll
    for (int h = (col + 1) / 2; h < 5; ++h) {
      const double2 v = C[col * 5 + h];
      if (2 * h > col) x[2 * h] -= v.x * x[col];
      x[2 * h + 1] -= v.y * x[col];
    }
  }
#pragma unroll
  for (int col = 9; col >= 0; --col) {
    double2 v[5];
#pragma unroll
    for (int h = 0; h <= col / 2; ++h) v[h] = C[col * 5 + h];
    x[col] *= (col & 1) ? v[col / 2].y : v[col / 2].x;
#pragma unroll
    for (int r = 0; r < col; ++r) x[r] -= ((r & 1) ? v[r / 2].y : v[r / 2].x) * x[col];
  }
}

// ten consecutive doubles of a thread
__device__ __forceinline__ void load10(const double* g, double (&v)[10]) {
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
#pragma unroll
    for (int h = 0; h < 5; ++h) {
      const double2 q = reinterpret_cast<const double2*>(g)[h];
      v[2 * h] = q.x;
      v[2 * h + 1] = q.y;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 10; ++e) v[e] = g[e];
  }
}
__device__ __forceinline__ void store10(double* g, const double (&v)[10]) {
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
#pragma unroll
    for (int h = 0; h < 5; ++h)
      reinterpret_cast<double2*>(g)[h] = make_double2(v[2 * h], v[2 * h + 1]);
  } else {
#pragma unroll
    for (int e = 0; e < 10; ++e) g[e] = v[e];
  }
}

__global__ void __launch_bounds__(kLuThreads, 8) block_lu_factor_kernel(long nb, double* A,
                                                                        int* __restrict__ piv,
                                                                        int* __restrict__ info_out) {
  extern __shared__ __align__(16) double sh[];  // [kLuThreads][kLuStride]
  int bad = 0;
  for (long blk0 = (long)blockIdx.x * kLuThreads; blk0 < nb; blk0 += (long)gridDim.x * kLuThreads) {
    const int nb_here = (int)((nb - blk0) < kLuThreads ? (nb - blk0) : kLuThreads);
    tile_in_async(A, sh, blk0, nb_here);
    tile_in_wait();
    if (threadIdx.x < nb_here) {
      double a[100];
      int p[10];
      double* mine = sh + threadIdx.x * kLuStride;
      double2* const m2 = reinterpret_cast<double2*>(mine);
#pragma unroll
      for (int e = 0; e < 50; ++e) {
        const double2 q = m2[e];
        a[2 * e] = q.x;
        a[2 * e + 1] = q.y;
      }
      if (lu10_regs(a, p)) bad = 1;
#pragma unroll
      for (int e = 0; e < 50; ++e) m2[e] = make_double2(a[2 * e], a[2 * e + 1]);
      int* pg = piv + (blk0 + threadIdx.x) * 10;
#pragma unroll
      for (int e = 0; e < 10; ++e) pg[e] = p[e];
    }
    __syncwarp();
    tile_out(A, sh, blk0, nb_here);
    __syncwarp();
  }
  if (bad) atomicMax(info_out, 1);
}

// Two tiles: the next one's copies, right-hand sides and pivots are in flight while this one is
// solved.  One warp a scheduler can keep the FP64 pipe busy by itself (an instruction's latency is
// its issue interval), so four such CTAs per SM do better than seven with one tile each, as long
// as little else is issued (192,000 blocks: 62 us with seven one-tile CTAs, 58 here).
__global__ void __launch_bounds__(kLuThreads) block_lu_solve_kernel(long nb,
                                                                    const double* __restrict__ LU,
                                                                    const int* __restrict__ piv,
                                                                    const double* b, double* x) {
  extern __shared__ __align__(16) double sh[];  // two LU tiles
  const long step = (long)gridDim.x * kLuThreads;
  double v[10];
  int p[10];
  auto fetch = [&](long at, double* tile) {
    const int m = (int)((nb - at) < kLuThreads ? (nb - at) : kLuThreads);
    tile_in_async(LU, tile, at, m);
    const long i = at + (threadIdx.x < m ? threadIdx.x : 0);
    load10(b + i * 10, v);
#pragma unroll
    for (int e = 0; e < 10; ++e) p[e] = __ldg(piv + i * 10 + e);
  };
  long blk0 = (long)blockIdx.x * kLuThreads;
  if (blk0 < nb) fetch(blk0, sh);
  for (int buf = 0; blk0 < nb; blk0 += step, buf ^= 1) {
    double now[10];
    int piv_now[10];
#pragma unroll
    for (int e = 0; e < 10; ++e) {
      now[e] = v[e];
      piv_now[e] = p[e];
    }
    tile_in_wait();
    if (blk0 + step < nb) fetch(blk0 + step, sh + (buf ^ 1) * (kLuThreads * kLuStride));
    if (blk0 + threadIdx.x < nb) {
      lus10(sh + buf * (kLuThreads * kLuStride) + threadIdx.x * kLuStride, piv_now, now);
      store10(x + (blk0 + threadIdx.x) * 10, now);
    }
    __syncwarp();
  }
}

// SUNMatScaleAddI(-gamma, J): A = -gamma*J + I on every block.  One fused multiply-add per
// element: adding -0 off the diagonal leaves the product as it is.  (A product and a predicated
// addition issued two FP64 instructions per warp for the three diagonal lanes in it.)
__device__ __forceinline__ double form_newton(double c, double v, int r) {
  return fma(c, v, (r % 11 == 0) ? 1.0 : -0.0);
}
template <bool PAIRS>
__global__ void block_form_newton_kernel(long nel, double* __restrict__ J, double c) {
  const long step = (long)gridDim.x * blockDim.x;
  if (PAIRS) {
    double2* const J2 = reinterpret_cast<double2*>(J);
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < nel / 2; e += step) {
      const int r = 2 * (int)((unsigned long)e % 50u);
      const double2 v = J2[e];
      J2[e] = make_double2(form_newton(c, v.x, r), form_newton(c, v.y, r + 1));
    }
  } else {
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < nel; e += step)
      J[e] = form_newton(c, J[e], (int)(e % 100));
  }
}

// persistent grid: as many CTAs as are resident (a few more would run alone at the end)
static int lu_grid(long nb, int per_sm) {
  long b = (nb + kLuThreads - 1) / kLuThreads;
  const long cap = (long)kSM * per_sm;
  if (b < 1) b = 1;
  return (int)(b < cap ? b : cap);
}

int block_lu_factor(long nb, double* A, int* piv, int* d_info, cudaStream_t s) {
  const size_t shm = sizeof(double) * kLuStride * kLuThreads;
  GBMV_CUDA_TRY(cudaFuncSetAttribute(block_lu_factor_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  ProfScope ps("block_lu_factor", s);
  block_lu_factor_kernel<<<lu_grid(nb, 8), kLuThreads, shm, s>>>(nb, A, piv, d_info);
  GBMV_LAUNCH_CHECK("block_lu_factor_kernel");
  return GBMV_OK;
}

int block_lu_solve(long nb, const double* LU, const int* piv, const double* b, double* x,
                   cudaStream_t s) {
  const size_t shm = sizeof(double) * 2 * kLuStride * kLuThreads;
  GBMV_CUDA_TRY(cudaFuncSetAttribute(block_lu_solve_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  ProfScope ps("block_lu_solve", s);
  block_lu_solve_kernel<<<lu_grid(nb, 4), kLuThreads, shm, s>>>(nb, LU, piv, b, x);
  GBMV_LAUNCH_CHECK("block_lu_solve_kernel");
  return GBMV_OK;
}

int block_form_newton(long nb, double* J, double gamma, cudaStream_t s) {
  const long nel = 100 * nb;
  const bool pairs = (reinterpret_cast<uintptr_t>(J) & 15) == 0;
  long g = ((pairs ? nel / 2 : nel) + 255) / 256;
  if (g > (long)kSM * 32) g = (long)kSM * 32;
  if (g < 1) g = 1;
  ProfScope ps("glue", s);
  if (pairs) block_form_newton_kernel<true><<<(int)g, 256, 0, s>>>(nel, J, -gamma);
  else block_form_newton_kernel<false><<<(int)g, 256, 0, s>>>(nel, J, -gamma);
  GBMV_LAUNCH_CHECK("block_form_newton_kernel");
  return GBMV_OK;
}

}  // namespace gbmv
