// bf16 "planes" of an FP64 matrix for the split-BF16 tensor-core GEMMs
// (oa_tgemm.cu): x = P_0 + P_1 (+ P_2), P_0 = bf16(x), P_1 = bf16(x - P_0),
// ..., stored in 64-column chunks, P[q][ldp / 64][rows_pad][64], so that a
// tile of 64 columns and any run of rows is one contiguous piece of memory.
// Kernels that produce such a matrix in FP64 can write its planes in the
// same pass (OaPlaneOut); the digits are the ones k_split_kc computes.
#pragma once
#include <cuda_bf16.h>

struct OaPlaneOut {
  void* P;        // bf16 planes, nullptr = none
  int rows_pad;   // rows per plane
  long ldp;       // leading size (a multiple of 64)
  int nt;         // planes: 2 or 3
};

// offset of element (r, c) in a plane of rows_pad rows
__host__ __device__ __forceinline__ size_t oa_plane_at(int r, long c, int rows_pad) {
  return ((size_t)(c >> 6) * rows_pad + r) * 64 + (size_t)(c & 63);
}

// a + b = s + e exactly, s = fl(a + b), for a = 0 or |a| >= |b| (Dekker's
// fast two-sum).  Here a is a remainder of the FP32 part, a multiple of its
// last place, and b the low part, at most half of that place.
__host__ __device__ __forceinline__ void oa_two_sum(float a, float b, float& s, float& e) {
  const float c = a + b;
  e = b - (c - a);
  s = c;
}

// the nt bf16 digits of v (nt <= 3): v is split into two FP32 parts first and
// the digits are taken in FP32 (conversions from and to FP64 run at a quarter
// of the FP32 rate); remainders are exact, so the digits are those of FP64
// remainders but for the low part's own rounding, 2^-48 below v
__host__ __device__ __forceinline__ void oa_bf16_digits(double v, int nt, __nv_bfloat16* h) {
  float r = (float)v, e = 0.f;
  const float lo = (float)(v - (double)r);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q >= nt) break;
    const __nv_bfloat16 b = __float2bfloat16_rn(r);
    h[q] = b;
    r -= __bfloat162float(b);
    if (q == 0) oa_two_sum(r, lo, r, e);
    else r += e;
  }
}

// the digits of a pair, one conversion instruction for both
__host__ __device__ __forceinline__ void oa_bf16_digits2(double x, double y, int nt, __nv_bfloat162* h) {
  float rx = (float)x, ry = (float)y, ex = 0.f, ey = 0.f;
  const float lx = (float)(x - (double)rx), ly = (float)(y - (double)ry);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q >= nt) break;
    const __nv_bfloat162 b = __floats2bfloat162_rn(rx, ry);
    h[q] = b;
    rx -= __low2float(b);
    ry -= __high2float(b);
    if (q == 0) {
      oa_two_sum(rx, lx, rx, ex);
      oa_two_sum(ry, ly, ry, ey);
    } else {
      rx += ex;
      ry += ey;
    }
  }
}

// planes of the element (r, c)
__device__ __forceinline__ void oa_plane_put(const OaPlaneOut& po, int r, long c, double x) {
  __nv_bfloat16 h[3];
  oa_bf16_digits(x, po.nt, h);
  __nv_bfloat16* base = (__nv_bfloat16*)po.P + oa_plane_at(r, c, po.rows_pad);
  const size_t pstride = (size_t)po.rows_pad * po.ldp;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q >= po.nt) break;
    base[q * pstride] = h[q];
  }
}

// planes of the pair (x, y) at row r, columns c and c + 1 (c even)
__device__ __forceinline__ void oa_plane_put2(const OaPlaneOut& po, int r, long c, double x, double y) {
  __nv_bfloat162 h[3];
  oa_bf16_digits2(x, y, po.nt, h);
  const unsigned cu = (unsigned)c;  // a row has fewer than 2^32 columns
  __nv_bfloat16* base =
      (__nv_bfloat16*)po.P + ((size_t)(cu >> 6) * (unsigned)po.rows_pad + (unsigned)r) * 64 + (cu & 63u);
  const size_t pstride = (size_t)po.rows_pad * po.ldp;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q >= po.nt) break;
    *reinterpret_cast<__nv_bfloat162*>(base + q * pstride) = h[q];
  }
}
