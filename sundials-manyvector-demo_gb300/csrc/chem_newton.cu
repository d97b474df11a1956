// Fused chemistry Newton step (parts b + c in one kernel): for every cell
//   f = TimeUnits * f_chem(y)                      (calculate_rhs_cvklu + N_VScale)
//   J = TimeUnits * df_chem/dy                     (calculate_jacobian_cvklu + scaling)
//   x = (I - gamma J)^{-1} f                       (SUNMatScaleAddI + getrf/getrs)
// without writing J to HBM.  One thread per cell; the cell's FP64 Newton matrix lives in a
// per-thread slice of shared memory ([element][thread], conflict-free).
//   LU = double: factor and solve in FP64 (the plain form fused);
//   LU = float : factor in FP32, solve in FP32, then `refine` steps of iterative refinement
//                with FP64 residuals r = f - A x against the FP64 matrix (the
//                mixed-precision Newton solve); a non-finite FP32 factor falls back to FP64.
// The temperature state (Ts, dTs/dge) is updated as by gbmv_chem_rhs (LU = double: exactly;
// LU = float: the ten Newton iterations run 8 in FP32 and the last 2 in FP64).
#include "chem.cuh"
#include "chem_net.cuh"
#include "chem_lu.cuh"
#include "df64.cuh"

namespace gbmv {

// Casts to and from the factor's precision, off the FP64 pipe (60 of a cell's ~900 FP64-pipe
// instructions were conversions; 96^3 cells 1751 -> 1683 us)
__device__ __forceinline__ double lu_cast(double x, double*) { return x; }
__device__ __forceinline__ float lu_cast(double x, float*) { return f32_of_f64<true>(x); }
__device__ __forceinline__ double lu_back(double x) { return x; }
__device__ __forceinline__ double lu_back(float x) { return f64_of_f32<true>(x); }

// Threads per block.  Shared memory per cell: the FP32-LU form keeps the 64 structural
// nonzeros of the FP64 Newton matrix (for the refinement residuals) and the variables, 592 bytes; the FP64-LU form
// its 100 entries until they are factored.  With 32-thread blocks eight fit an SM, the register
// limit.
constexpr int kNtThreads = 32;

// The cell's scaled variables are kept in its shared-memory slice (f may be written over y):
// after the FP64 matrix entries in the FP32-LU form, in ten places of the FP64 form's matrix
// that are structurally zero (column-major rows 4-8 of column 0, 5-7 and 9 of column 1, 5 of 2).
__device__ constexpr int kZeroSlot[10] = {4, 5, 6, 7, 8, 15, 16, 17, 19, 25};
template <typename LU>
__device__ __forceinline__ constexpr int z_slot(int s) {
  return sizeof(LU) == 4 ? 64 + s : kZeroSlot[s];
}

// entry (row, col) of the Newton matrix: FP32-LU form to the FP64 pattern, FP64 form to the factor
template <typename LU, int BS>
__device__ __forceinline__ void put_entry(double* As, LU* L, int row, int col, double a) {
  if (sizeof(LU) == 4) {
    const int e = kJacIndex[row][col];
    if (e >= 0) As[e * BS] = a;
  } else {
    L[(col * 10 + row) * BS] = to_lu<LU>(a);
  }
}

// The Newton matrix without the column scaling (a rare path): every entry from its own expression
template <typename LU, int BS>
static __device__ __noinline__ void newton_matrix_plain(const ChemParams& P, const ChemState& S,
                                                        long i, double T, double dT, double gt,
                                                        double* As, LU* L) {
  const long j = i * 10;
  double ya[10], pr[21], k[kNRates], dk[kNRates];
#pragma unroll
  for (int s = 0; s < 10; ++s) ya[s] = As[z_slot<LU>(s) * BS] * S.scale[j + s];
  chem_rates<true>(P, chem_log(P, T), k, dk);
  chem_products(ya, pr);
  const ChemAux A{S.mdens[i], S.imdens[i], S.cie[i], S.h2[i]};
  chem_jacobian(P, k, dk, ya, pr, T, dT * (P.idbin * rcp64_any(T)), A, ge_terms(k, ya),
                [&](int row, int col, double v) {
                  put_entry<LU, BS>(As, L, row, col,
                                    (v * (-gt * S.inv_scale[j + row])) * S.scale[j + col] +
                                        (row == col ? 1.0 : 0.0));
                });
}

template <typename LU, int BS>
__global__ void __launch_bounds__(BS) chem_newton_kernel(ChemParams P, ChemState S, long n,
                                                         const double* __restrict__ y,
                                                         double* __restrict__ fout,
                                                         double* __restrict__ xout,
                                                         double gamma, double tunit,
                                                         int refine,
                                                         int* __restrict__ info_out,
                                                         const double* __restrict__ bst,
                                                         unsigned long long* __restrict__ queue) {
  extern __shared__ unsigned char smem_raw[];
  constexpr bool kMixed = sizeof(LU) == 4;
  // variables whose columns are scaled by them: 2^-kRange to 2^kRange.  FP32 entries take products
  // of two such scales with the matrix' own range and stay in the float range (at 2^+-99, variables
  // over 56 decades and no refinement, the median cell lost every digit; plain 3e-4)
  constexpr unsigned kRange = kMixed ? 40 : 99;
  // FP32-LU form: As[e * BS] = FP64 matrix entry e of kJacPattern; FP64 form: L[(col*10+row) * BS]
  double* As = reinterpret_cast<double*>(smem_raw) + threadIdx.x;
  LU* L = reinterpret_cast<LU*>(smem_raw) + threadIdx.x;
  int bad = 0;
  // cells: a grid-stride sweep, or (queue set) 32-cell chunks taken from the shared counter by
  // each one-warp block until every cell is taken (launches on other streams may share it)
  long i = queue ? -1 : blockIdx.x * (long)blockDim.x + threadIdx.x;
  const long stride = (long)gridDim.x * blockDim.x;
  while (true) {
    if (queue) {
      unsigned long long base = 0;
      if (threadIdx.x == 0) base = atomicAdd(queue, (unsigned long long)BS);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= (unsigned long long)n) break;
      i = (long)base + threadIdx.x;
    } else if (i >= n) {
      break;
    }
    if (i < n) {  // (the last chunk's surplus lanes skip the cell and take the next, empty one)
      const long j = i * 10;
      const double* __restrict__ sc = S.scale + j;  // re-read through L1: keeps registers free
      const double* __restrict__ isc = S.inv_scale + j;
      double ya[10];
      bool scaled = true;  // see below
#pragma unroll
      for (int s = 0; s < 10; ++s) {
        const double z = y[j + s];
        ya[s] = z * sc[s];
        As[z_slot<LU>(s) * BS] = z;
        const int e = (__double2hiint(z) >> 20) & 0x7FF;
        scaled = scaled && (unsigned)(e - (1023 - kRange)) <= 2u * kRange;
      }
      double Ts = S.Ts[i], dTs = 0.0, logT;
      // mixed form: up to 8 FP32 iterations, then two in FP64.  (One FP64 iteration where
      // the FP32 stage converged measured 5 % faster but left the carried temperature up to
      // 4e-10 off the FP64 form's ten-iteration value: the adiabatic-index tables are linear
      // in log T per bin, so near a bin edge Newton converges only linearly.)
      if (sizeof(LU) == 4)
        chem_temperature_mixed(P, ya, Ts, dTs, logT, 8);
      else
        chem_temperature(P, ya, Ts, dTs, logT);
      S.Ts[i] = Ts;
      S.dTs_ge[i] = dTs;
      const ChemAux Ax{S.mdens[i], S.imdens[i], S.cie[i], S.h2[i]};
      double f[10];
      // The matrix is formed with every column multiplied by its own variable, A diag(z): its
      // species entries are then plain sums of the reaction fluxes (chem_matrix), and partial
      // pivoting, which compares within a column, picks the same rows.  The solution is z times
      // that system's.  Variables that are zero or far from 1 (kRange) take the unscaled matrix.
      {  // source and Newton matrix from one rate evaluation (rates and T slopes)
        double k[kNRates], dk[kNRates], pr[21], r[21];
        chem_rates<true>(P, logT, k, dk);
        const GeTerms Rg = ge_terms(k, ya);  // shared by the source and the Jacobian's ge row
        chem_products(ya, pr);
        chem_fluxes(k, pr, r);
        {
          double sp[9];
          chem_species(r, sp);
#pragma unroll
          for (int s = 0; s < 9; ++s) f[s] = (sp[s] * isc[s]) * tunit;
          double ge = chem_ge_source(P, k, ya, Ts, Ax, Rg) * isc[9];
          ge *= Ax.imdens;
          f[9] = ge * tunit;
        }
#pragma unroll
        for (int s = 0; s < 10; ++s) fout[j + s] = f[s];
        if (scaled) {
          double rf[10];  // -gamma * tunit * inv_scale[row], the ge row's 1/mdensity with it
#pragma unroll
          for (int q = 0; q < 10; ++q) rf[q] = (-gamma * tunit) * isc[q];
          rf[9] *= Ax.imdens;
          const double t9 = dTs * (P.idbin * rcp64_any(Ts)) * ya[9];
          // every structural entry (the diagonal included) is put exactly once
          chem_matrix(P, k, dk, ya, pr, r, Ts, Ax, Rg, [&](int row, int col, double v) {
            const double u = col == 9 ? v * t9 : v;
            put_entry<LU, BS>(As, L, row, col, row == col ? fma(u, rf[row], As[z_slot<LU>(row) * BS]) : u * rf[row]);
          });
        } else {
          newton_matrix_plain<LU, BS>(P, S, i, Ts, dTs, gamma * tunit, As, L);
        }
      }
#pragma unroll
      for (int s = 0; s < 10; ++s) f[s] = fout[j + s];
      if (bst) {  // implicit-stage form: right-hand side b + gamma f(y)
#pragma unroll
        for (int s = 0; s < 10; ++s) f[s] = fma(gamma, f[s], bst[j + s]);
      }

      int piv[10];
      double x[10];
      // (Power-of-two row, or row and column, equilibration of the FP32 factor was tried: on
      // these matrices it changes the pivot order for the worse -- 2.4e-3 against 1.9e-8 after
      // one refinement on the test blocks, reproduced on the oracle's matrices -- so the factor
      // keeps plain partial pivoting.)
      float zf[10];  // z for the stopping tests, which are on x
      if (sizeof(LU) == 4) {
#pragma unroll
        for (int s = 0; s < 10; ++s) zf[s] = scaled ? f32_of_f64(As[z_slot<LU>(s) * BS]) : 1.f;
      }
      // the factor lives in registers: in shared memory every elimination step waited on its
      // loads (7-8 warps per SM); FP32 entries converted with integer instructions
      LU a[100];
#pragma unroll
      for (int e = 0; e < 100; ++e) {
        const int q = kJacIndex[e % 10][e / 10];
        if (q < 0) a[e] = LU(0);  // structural zero
        else if constexpr (kMixed) a[e] = f32_of_f64(As[q * BS]);
        else a[e] = L[e * BS];
      }
      int info = lu10_regs(a, piv);
      bool fp64_fallback = (sizeof(LU) == 4) && info != 0;
      if (!fp64_fallback) {
        LU xs[10];
#pragma unroll
        for (int s = 0; s < 10; ++s) xs[s] = lu_cast(f[s], (LU*)nullptr);
        lus10_regs(a, piv, xs);
        float xmax = 0.f;  // solution size for the stopping tests, from the FP32 solve: the
                           // refinements move it by ~1e-7 relative, far below either threshold
#pragma unroll
        for (int s = 0; s < 10; ++s) {
          x[s] = lu_back(xs[s]);
          if (kMixed) xmax = fmaxf(xmax, fabsf((float)xs[s] * zf[s]));
        }
        if (sizeof(LU) == 4) {
          // iterative refinement against FP64 residuals; a cell stops as soon as its correction
          // is below 1e-13 of the solution (well-conditioned cells need one step, the
          // ill-conditioned ones use up to `refine`); a cell whose last correction is still above
          // 1e-6 of its solution (the FP32 factor too poor a preconditioner for its block)
          // takes the FP64 factor below
          float dlast = 0.f;
          for (int it = 0; it < refine; ++it) {
            double rr[10];
#pragma unroll
            for (int row = 0; row < 10; ++row) rr[row] = f[row];
#pragma unroll
            for (int e = 0; e < 64; ++e)  // the 64 structural nonzeros (diagonal included)
              rr[kJacPattern[e][0]] -= As[e * BS] * x[kJacPattern[e][1]];
            LU ds[10];
#pragma unroll
            for (int s = 0; s < 10; ++s) ds[s] = lu_cast(rr[s], (LU*)nullptr);
            lus10_regs(a, piv, ds);
            float dmax = 0.f;
#pragma unroll
            for (int s = 0; s < 10; ++s) {
              x[s] += lu_back(ds[s]);
              dmax = fmaxf(dmax, fabsf((float)ds[s] * zf[s]));
            }
            dlast = dmax;
            if (dmax <= 1e-13f * xmax) break;
          }
          bool finite = true;
#pragma unroll
          for (int s = 0; s < 10; ++s) finite = finite && isfinite(x[s]);
          fp64_fallback = !finite || !(dlast <= 1e-6f * xmax);
        }
      }
      if (fp64_fallback) {  // FP32 factor singular or out of range: factor the FP64 matrix,
                            // rebuilt densely in (per-thread local) memory -- a rare path
        double Ad[100];
        for (int e = 0; e < 100; ++e) Ad[e] = 0.0;
        for (int e = 0; e < 64; ++e) Ad[kJacPattern[e][1] * 10 + kJacPattern[e][0]] = As[e * BS];
        info = lu10_strided<double, true>(Ad, 1, piv);
#pragma unroll
        for (int s = 0; s < 10; ++s) x[s] = f[s];
        lus10_strided<double, double>(Ad, 1, piv, x);
      }
      if (info && (sizeof(LU) == 8 || fp64_fallback)) bad = 1;
#pragma unroll
      for (int s = 0; s < 10; ++s) xout[j + s] = scaled ? x[s] * As[z_slot<LU>(s) * BS] : x[s];
    }
    if (!queue) i += stride;
  }
  if (bad) atomicMax(info_out, 1);
}

template <typename LU>
static int launch_newton(const ChemParams& P, const ChemState& S, long n, const double* y,
                         double* f, double* x, double gamma, double tunit, int refine,
                         int* d_info, cudaStream_t s, long blocks, const double* b,
                         unsigned long long* queue) {
  constexpr int BS = kNtThreads;
  const size_t shm = (size_t)BS * (sizeof(LU) == 4 ? 74 : 100) * sizeof(double);
  // a function attribute, not a stream operation: also legal during graph capture
  GBMV_CUDA_TRY(cudaFuncSetAttribute(chem_newton_kernel<LU, BS>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  chem_newton_kernel<LU, BS><<<(int)blocks, BS, shm, s>>>(P, S, n, y, f, x, gamma, tunit,
                                                          refine, d_info, b, queue);
  GBMV_LAUNCH_CHECK("chem_newton_kernel");
  return GBMV_OK;
}

int chem_newton(const ChemParams& P, const ChemState& S, long n, const double* y, double* f,
                double* x, double gamma, double tunit, int lu_fp32, int refine, int* d_info,
                cudaStream_t s, int blocks_per_sm, const double* b,
                unsigned long long* queue) {
  long blk = (n + kNtThreads - 1) / kNtThreads;
  // default: a deep grid-stride grid; blocks_per_sm > 0: exactly that many resident blocks per
  // SM (a persistent grid leaving room for a kernel running beside it on another stream)
  const long cap = (long)kSM * (blocks_per_sm > 0 ? blocks_per_sm : 48);
  if (blk > cap) blk = cap;
  if (blk < 1) blk = 1;
  ProfScope ps("chem_newton", s);
  if (lu_fp32)
    return launch_newton<float>(P, S, n, y, f, x, gamma, tunit, refine, d_info, s, blk, b,
                                queue);
  return launch_newton<double>(P, S, n, y, f, x, gamma, tunit, refine, d_info, s, blk, b,
                               queue);
}

}  // namespace gbmv
