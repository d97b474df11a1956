// Tiles of 32 consecutive 10x10 blocks between global and shared memory, for kernels whose CTA is
// one warp with a block per thread (blocklu.cu, the Jacobian of chem.cu).
#pragma once

#include "common.cuh"

namespace gbmv {

constexpr int kLuThreads = 32;   // blocks per tile = threads per CTA
constexpr int kLuStride = 102;   // per-block stride of the shared tile (doubles): a multiple of 16
                                 // bytes, and two-way bank conflicts at most

// Copy of `nb` consecutive blocks of 100 doubles into the shared tile; waits for nothing.
// 16-byte asynchronous copies where the address allows (caller arrays need only be 8-byte
// aligned).  A full tile goes block by block, a chunk a lane, so that every address is the
// lane's plus a constant: dividing a running chunk number cost more issue slots than the solve's
// arithmetic left free.
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void tile_in_async(const double* __restrict__ g, double* sh, long blk0,
                                              int nb) {
  const double* src = g + blk0 * 100;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const unsigned base = (unsigned)__cvta_generic_to_shared(sh);
    const int lane = threadIdx.x;
    if (nb == kLuThreads) {
      const unsigned d = base + 16 * lane;
      const double* const q = src + 2 * lane;
#pragma unroll
      for (int k = 0; k < kLuThreads; ++k) cp_async16(d + k * (kLuStride * 8), q + k * 100);
      if (lane < 18) {
#pragma unroll
        for (int k = 0; k < kLuThreads; ++k)
          cp_async16(d + k * (kLuStride * 8) + 512, q + k * 100 + 64);
      }
    } else {
      for (int c = lane; c < nb * 50; c += kLuThreads)
        cp_async16(base + (unsigned)((c / 50) * (kLuStride * 8) + (c % 50) * 16), src + 2 * c);
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
    const int lane = threadIdx.x;
    if (nb == kLuThreads) {
      const double2* const s = reinterpret_cast<const double2*>(sh) + lane;
      double2* const d = reinterpret_cast<double2*>(dst) + lane;
#pragma unroll 8
      for (int k = 0; k < kLuThreads; ++k) d[k * 50] = s[k * (kLuStride / 2)];
      if (lane < 18) {
#pragma unroll 8
        for (int k = 0; k < kLuThreads; ++k) d[k * 50 + 32] = s[k * (kLuStride / 2) + 32];
      }
    } else {
      for (int c = lane; c < nb * 50; c += kLuThreads)
        reinterpret_cast<double2*>(dst)[c] =
            *reinterpret_cast<const double2*>(sh + (c / 50) * kLuStride + 2 * (c % 50));
    }
  } else {
    for (int c = threadIdx.x; c < nb * 100; c += kLuThreads)
      dst[c] = sh[(c / 100) * kLuStride + c % 100];
  }
}

}  // namespace gbmv
