// Helpers of the density kernels.
#pragma once
#include "oa_internal.h"

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block sum of NV doubles; results in out[] of thread 0
template <int NV>
__device__ void block_sum_n(double* v, double* sh /* 32*NV */) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = warp_sum_d(v[k]);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k * 32 + wid] = v[k];
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double r = (lane < nw) ? sh[k * 32 + lane] : 0.0;
      v[k] = warp_sum_d(r);
    }
  }
}

__host__ __device__ static inline size_t align_up_r(size_t x, size_t a) { return (x + a - 1) / a * a; }

// 16-byte global -> shared copy without a register round trip, so that a
// block's staging copies are all in flight together (the caller commits
// the group and waits for it)
__device__ __forceinline__ void rho_cp16(void* sdst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc));
}
__device__ __forceinline__ void rho_cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void rho_cp_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
