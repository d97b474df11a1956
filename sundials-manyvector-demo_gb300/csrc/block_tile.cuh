// Tiles of 32 consecutive 10x10 blocks between global and shared memory, for kernels whose CTA is
// one warp with a block per thread (blocklu.cu, the Jacobian of chem.cu).
#pragma once

#include "common.cuh"

namespace gbmv {

constexpr int kLuThreads = 32;   // blocks per tile = threads per CTA
constexpr int kLuStride = 102;   // per-block stride of the shared tile (doubles): a multiple of 16
                                 // bytes, and two-way bank conflicts at most
constexpr int kVecStride = 11;   // the same for the right-hand-side tile

// Copy of `nb` consecutive blocks of 100 doubles into the shared tile; waits for nothing.
// 16-byte asynchronous copies where the address allows (caller arrays need only be 8-byte
// aligned).
__device__ __forceinline__ void tile_in_async(const double* __restrict__ g, double* sh, long blk0,
                                              int nb) {
  const double* src = g + blk0 * 100;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const unsigned base = (unsigned)__cvta_generic_to_shared(sh);
#pragma unroll 10
    for (int c = threadIdx.x; c < nb * 50; c += kLuThreads) {
      const int b = c / 50, e = c - b * 50;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       base + (unsigned)(b * (kLuStride * 8) + e * 16)),
                   "l"(src + 2 * c)
                   : "memory");
    }
  } else {
    for (int c = threadIdx.x; c < nb * 100; c += kLuThreads)
      sh[(c / 100) * kLuStride + c % 100] = src[c];
  }
}
__device__ __forceinline__ void tile_in_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void tile_out(double* __restrict__ g, const double* sh, long blk0,
                                         int nb) {
  double* dst = g + blk0 * 100;
  if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll 10
    for (int c = threadIdx.x; c < nb * 50; c += kLuThreads) {
      const int b = c / 50, e = c - b * 50;
      reinterpret_cast<double2*>(dst)[c] =
          *reinterpret_cast<const double2*>(sh + b * kLuStride + 2 * e);
    }
  } else {
    for (int c = threadIdx.x; c < nb * 100; c += kLuThreads)
      dst[c] = sh[(c / 100) * kLuStride + c % 100];
  }
}

}  // namespace gbmv
