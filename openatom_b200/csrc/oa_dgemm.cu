// Pipelined FP64 tensor-core (DMMA) forward product of the PairCalculator:
//   C[i][j] = alpha sum_k w(k) A[i][k] B[j][k],  w(k) = w_kx0 for k < kx0_cols, else 1
// (PairCalculator::multiplyForward, ckPairCalculator.C:821-933, with the
// reference's DGEMM('T','N') on the 2*ng-double real view of each state).
//
// Split-K over slabs of 32 columns: the kx0 columns [0, kx0_cols) are shared
// out among the first n0 CTAs of a tile and the other columns among the
// remaining nr CTAs, slab t of a region going to CTA t mod (count), so at
// any moment the CTAs stream neighbouring 256-byte pieces of the same rows
// (DRAM pages are opened once, not once per CTA).  Each CTA writes an FP64
// partial of its 128 x 128 output tile; the kx0 weight is applied to the
// first n0 partials in the reduction, so the main loop has no per-column
// weight and, when A and B are the same matrix (the overlap S), one shared
// memory copy of the operand slab serves both sides.  Partials are summed in
// a fixed order: the result does not depend on scheduling.
//
// Main loop: 512 threads, 16 warps of 32 x 32 (4 x 4 DMMA m8n8k4 tiles); K
// slabs of 32 doubles move global -> shared with 16-byte cp.async into a
// ring of STAGES slabs (4 when A and B are one matrix, else 3: 144 / 216 KB),
// so the loads of the next slabs overlap the DMMAs of the current one.
#include <algorithm>
#include "oa_internal.h"

#define DG_TM 128
#define DG_KS 32
#define DG_LD (DG_KS + 4)          // doubles per smem row: conflict-free fragment loads
#define DG_THREADS 512
#define DG_SLAB (DG_TM * DG_LD)    // doubles per operand slab

__device__ __forceinline__ void dg_dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}

__device__ __forceinline__ void dg_cp16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;  // src-size 0: the 16 bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void dg_cp8(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void dg_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void dg_wait() { asm volatile("cp.async.wait_group %0;\n" :: "n"(N)); }

// one operand slab: rows [r0, r0 + 128) of X (row stride K), columns [k0, k0 + 32)
// clipped to [k0, kend) and rows < nrows; 2048 16-byte pieces, 4 per thread
__device__ __forceinline__ void dg_load_slab(double* dst, const double* __restrict__ X, int r0, int nrows, long K,
                                             long k0, long kend) {
#pragma unroll
  for (int q = 0; q < (DG_TM * DG_KS / 2) / DG_THREADS; ++q) {
    const int piece = threadIdx.x + q * DG_THREADS;
    const int r = piece >> 4;            // 16 pieces per row
    const int kk = (piece & 15) * 2;
    const long k = k0 + kk;
    const bool valid = (r0 + r < nrows) && (k < kend);
    const double* src = valid ? X + (size_t)(r0 + r) * K + k : X;
    dg_cp16(dst + r * DG_LD + kk, src, valid);
  }
}

// Output tiles of a product and the CTAs of each: tile t covers rows
// 128 ti .., columns 128 tj .. and owns the CTAs [start[t], start[t + 1]), the
// first n0[t] of them on the kx0 columns.  A tile's CTAs are in proportion to
// the DMMAs that its busiest SM sub-partition issues (edge tiles and the
// diagonal tiles of a symmetric product have fewer), so that all CTAs of the
// product take the same time: S of 199 states on three tiles, for instance,
// splits its SMs 59 : 44 : 44.
// nt = 0 (more than 8 row or column tiles): CTA row y of the grid is tile
// (y / tj[0], y mod tj[0]), all with the CTA counts of entry 0.
#define DG_MAXT 64
struct DgTiles {
  int nt, sym;
  short ti[DG_MAXT], tj[DG_MAXT], n0[DG_MAXT], start[DG_MAXT + 1];
  signed char at[8][8];  // tile of (row tile, column tile), -1: the mirror of a symmetric product
};

template <bool SAME, int DG_STAGES>
__global__ void __launch_bounds__(DG_THREADS, 1)
k_dgemm_fwd(const double* __restrict__ A, const double* __restrict__ B, int m, int n, long K, long kx0_cols,
            const __grid_constant__ DgTiles tiles, double* __restrict__ part, const int* __restrict__ cond) {
  if (cond && *cond == 0) return;
  extern __shared__ __align__(16) double dg_smem[];
  int t = 0;
  while (t + 1 < tiles.nt && (int)blockIdx.x >= tiles.start[t + 1]) ++t;
  const int i0 = (tiles.nt ? tiles.ti[t] : (int)blockIdx.y / tiles.tj[0]) * DG_TM;
  const int j0 = (tiles.nt ? tiles.tj[t] : (int)blockIdx.y % tiles.tj[0]) * DG_TM;
  const int kb = blockIdx.x - tiles.start[t];
  const int n0 = tiles.n0[t], nr = tiles.start[t + 1] - tiles.start[t] - n0;
  // a diagonal tile of a symmetric product: one operand slab serves both sides
  const bool diag = SAME || (tiles.sym && i0 == j0);
  double* As = dg_smem;
  double* Bs = diag ? dg_smem : dg_smem + DG_STAGES * DG_SLAB;
  // region and slab sequence of this CTA: slabs first, first + stride, ...
  const bool in0 = kb < n0;
  const long rbeg = in0 ? 0 : kx0_cols, rend = in0 ? kx0_cols : K;
  const int first = in0 ? kb : kb - n0, stride = in0 ? n0 : nr;
  const long rslabs = (rend - rbeg + DG_KS - 1) / DG_KS;
  const int nslab = rslabs > first ? (int)((rslabs - first + stride - 1) / stride) : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Block (wi, wj) of a warp: the blocks of a row or column go to different
  // SM sub-partitions (warp mod 4), so that a tile with fewer than four block
  // rows or columns loads them evenly.  On a diagonal tile of a symmetric
  // product the 32 x 32 blocks below the diagonal are the transposes of those
  // above, which the reduction mirrors; the ten blocks on and above it go to
  // warps 0-9, at most three per sub-partition.
  int wi = (warp >> 2) * 32, wj = (((warp & 3) + (warp >> 2)) & 3) * 32;
  if (diag) {
    // 4 bi + bj of the upper blocks 0, 1, 2, 3, 5, 6, 7, 10, 11, 15, one hex digit per warp
    const int u = warp < 10 ? (int)((0xFBA7653210ull >> (4 * warp)) & 15u) : 0;
    wi = (u >> 2) * 32;
    wj = (u & 3) * 32;
  }
  const bool active = (i0 + wi < m) && (j0 + wj < n) && (!diag || warp < 10);
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) { acc[a][b][0] = 0.0; acc[a][b][1] = 0.0; }
  // prologue: slabs 0 .. STAGES-2
#pragma unroll
  for (int s = 0; s < DG_STAGES - 1; ++s) {
    if (s < nslab) {
      const long k0 = rbeg + ((long)first + (long)s * stride) * DG_KS;
      dg_load_slab(As + s * DG_SLAB, A, i0, m, K, k0, rend);
      if (!diag) dg_load_slab(Bs + s * DG_SLAB, B, j0, n, K, k0, rend);
    }
    dg_commit();
  }
  for (int s = 0; s < nslab; ++s) {
    dg_wait<DG_STAGES - 2>();
    __syncthreads();
    // refill the stage freed by slab s - 1
    {
      const int sn = s + DG_STAGES - 1;
      if (sn < nslab) {
        const int st = sn % DG_STAGES;
        const long k0 = rbeg + ((long)first + (long)sn * stride) * DG_KS;
        dg_load_slab(As + st * DG_SLAB, A, i0, m, K, k0, rend);
        if (!diag) dg_load_slab(Bs + st * DG_SLAB, B, j0, n, K, k0, rend);
      }
      dg_commit();
    }
    const double* as = As + (s % DG_STAGES) * DG_SLAB;
    const double* bs = Bs + (s % DG_STAGES) * DG_SLAB;
    if (active) {
#pragma unroll
      for (int k4 = 0; k4 < DG_KS; k4 += 4) {
        double af[4], bf[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) af[q] = as[(wi + q * 8 + (lane >> 2)) * DG_LD + k4 + (lane & 3)];
#pragma unroll
        for (int q = 0; q < 4; ++q) bf[q] = bs[(wj + q * 8 + (lane >> 2)) * DG_LD + k4 + (lane & 3)];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) dg_dmma(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
      }
    }
  }
  dg_wait<0>();
  if (!active) return;
  double* out = part + (size_t)kb * m * n;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = i0 + wi + a * 8 + (lane >> 2);
      const int j = j0 + wj + b * 8 + 2 * (lane & 3);
      if (i < m && j < n) out[(size_t)i * n + j] = acc[a][b][0];
      if (i < m && j + 1 < n) out[(size_t)i * n + j + 1] = acc[a][b][1];
    }
}

// C = alpha (w0 sum_{kb < n0} part[kb] + sum_{kb >= n0} part[kb]) over the
// partials of an output's tile; an output below the diagonal blocks of a
// symmetric product reads its transpose.  Block = 64 outputs x 4 partial groups (group g sums the partials kb = g mod 4 of
// each range); the groups are combined in a fixed order, so the result does
// not depend on scheduling.
#define DR_COLS 64
#define DR_GROUPS 4
__global__ void __launch_bounds__(DR_COLS * DR_GROUPS)
k_dgemm_fwd_reduce(const double* __restrict__ part, const __grid_constant__ DgTiles tiles, int n, size_t nn,
                   double w0, double alpha, double* __restrict__ C, const int* __restrict__ cond) {
  if (cond && *cond == 0) return;
  __shared__ double s0s[DR_GROUPS][DR_COLS], s1s[DR_GROUPS][DR_COLS];
  const int col = threadIdx.x % DR_COLS, g = threadIdx.x / DR_COLS;
  const size_t i = (size_t)blockIdx.x * DR_COLS + col;
  size_t src = i;
  int n0 = 0, nkb = 0;
  if (i < nn) {
    int r = (int)(i / n), c = (int)(i - (size_t)r * n);
    if (tiles.sym && (r >> 5) > (c >> 5)) {
      src = (size_t)c * n + r;
      const int s = r; r = c; c = s;
    }
    const int t = tiles.nt > 1 ? tiles.at[r >> 7][c >> 7] : 0;
    n0 = tiles.n0[t];
    nkb = tiles.start[t + 1] - tiles.start[t];
  }
  double s0 = 0.0, s1 = 0.0;
  if (i < nn) {
    for (int k = g; k < n0; k += DR_GROUPS) s0 += __ldcs(part + (size_t)k * nn + src);
    int k = n0 + g;
    for (; k + 3 * DR_GROUPS < nkb; k += 4 * DR_GROUPS) {
      const double a = __ldcs(part + (size_t)k * nn + src);
      const double b = __ldcs(part + (size_t)(k + DR_GROUPS) * nn + src);
      const double c = __ldcs(part + (size_t)(k + 2 * DR_GROUPS) * nn + src);
      const double d = __ldcs(part + (size_t)(k + 3 * DR_GROUPS) * nn + src);
      s1 += a; s1 += b; s1 += c; s1 += d;
    }
    for (; k < nkb; k += DR_GROUPS) s1 += __ldcs(part + (size_t)k * nn + src);
  }
  s0s[g][col] = s0;
  s1s[g][col] = s1;
  __syncthreads();
  if (g == 0 && i < nn) {
    double t0 = 0.0, t1 = 0.0;
#pragma unroll
    for (int q = 0; q < DR_GROUPS; ++q) { t0 += s0s[q][col]; t1 += s1s[q][col]; }
    C[i] = alpha * (w0 * t0 + t1);
  }
}

#define DG_STAGES_SAME 4
#define DG_STAGES_TWO 3
size_t oa_dgemm_fwd_smem(bool same) {
  return same ? (size_t)DG_STAGES_SAME * DG_SLAB * sizeof(double) : (size_t)2 * DG_STAGES_TWO * DG_SLAB * sizeof(double);
}

// Returns cudaErrorNotSupported when the operands do not allow 16-byte
// copies (odd K, odd kx0_cols or unaligned pointers); the caller then uses
// the element-wise kernel.  nkb bounds the partials the caller provides
// (part holds nkb * m * n doubles).
// cond: optional device flag; when it is 0 at run time the launches do nothing
// (the conditional PsiV reset of the native step).
cudaError_t oa_dgemm_fwd(cudaStream_t s, const double* A, const double* B, int m, int n, long K, long kx0_cols,
                         double w_kx0, double alpha, double* part, int nkb, double* C, const int* cond) {
  if ((K & 1) || (kx0_cols & 1) || (((uintptr_t)A | (uintptr_t)B) & 15) || kx0_cols > K || nkb < 2)
    return cudaErrorNotSupported;
  // SM count of the current device (per call: processes may drive GPUs of
  // different sizes)
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0)
    nsm = 148;
  const int ti = (m + DG_TM - 1) / DG_TM, tj = (n + DG_TM - 1) / DG_TM;
  const bool listed = ti <= 8 && tj <= 8;
  const bool sym = A == B && m == n && listed;
  DgTiles tiles;
  tiles.sym = sym;
  tiles.nt = 0;
  // DMMA load of a tile: blocks of its busiest sub-partition
  int load[DG_MAXT], total = 0;
  for (int a = 0; listed && a < ti; ++a)
    for (int b = 0; b < tj; ++b) {
      tiles.at[a][b] = -1;
      if (sym && b < a) continue;
      const int rb = (std::min(m - a * DG_TM, DG_TM) + 31) / 32, cb = (std::min(n - b * DG_TM, DG_TM) + 31) / 32;
      const int t = tiles.nt++;
      tiles.ti[t] = (short)a;
      tiles.tj[t] = (short)b;
      tiles.at[a][b] = (signed char)t;
      load[t] = sym && a == b ? (rb == 4 ? 3 : std::min(rb, 2)) : std::min(rb, cb);
      total += load[t];
    }
  if (!listed) {
    tiles.tj[0] = (short)tj;
    load[0] = 1;
    total = ti * tj;
  }
  // about one CTA per SM; the kx0 region gets CTAs in proportion to its slabs
  const long s0 = (kx0_cols + DG_KS - 1) / DG_KS, sr = (K - kx0_cols + DG_KS - 1) / DG_KS;
  int cta = 0;
  for (int t = 0; t < std::max(tiles.nt, 1); ++t) {
    int nk = (int)((long)nsm * load[t] / total);
    if (nk > nkb) nk = nkb;
    if (nk < 2) nk = 2;
    int n0 = s0 > 0 ? (int)((nk * s0 + s0 + sr - 1) / (s0 + sr)) : 0;  // rounded up: no straggler
    if (s0 > 0 && n0 < 1) n0 = 1;
    if (n0 > s0) n0 = (int)s0;
    int nr = nk - n0;
    if (nr > sr) nr = (int)sr;
    if (sr > 0 && nr < 1) return cudaErrorNotSupported;
    if (n0 + nr < 1 || n0 + nr > nkb) return cudaErrorNotSupported;
    tiles.n0[t] = (short)n0;
    tiles.start[t] = (short)cta;
    cta += n0 + nr;
    tiles.start[t + 1] = (short)cta;
  }
  const dim3 grid(cta, listed ? 1 : ti * tj);
  // one shared slab per stage when the single output tile is diagonal
  // (A == B, m = n <= 128)
  const bool same = sym && tiles.nt == 1;
  const size_t sm = oa_dgemm_fwd_smem(same);
  cudaError_t e;
  if (same) {
    e = oa_smem_limit(k_dgemm_fwd<true, DG_STAGES_SAME>);
    if (e != cudaSuccess) return e;
    k_dgemm_fwd<true, DG_STAGES_SAME><<<grid, DG_THREADS, sm, s>>>(A, B, m, n, K, kx0_cols, tiles, part, cond);
  } else {
    e = oa_smem_limit(k_dgemm_fwd<false, DG_STAGES_TWO>);
    if (e != cudaSuccess) return e;
    k_dgemm_fwd<false, DG_STAGES_TWO><<<grid, DG_THREADS, sm, s>>>(A, B, m, n, K, kx0_cols, tiles, part, cond);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const size_t mn = (size_t)m * n;
  k_dgemm_fwd_reduce<<<(unsigned)((mn + DR_COLS - 1) / DR_COLS), DR_COLS * DR_GROUPS, 0, s>>>(
      part, tiles, n, mn, w_kx0, alpha, C, cond);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Backward product (PairCalculator::multiplyResult / bwMultiplyHelper /
// bwMultiplyDynOrthoT, ckPairCalculator.C:1201-1468, 1710-2031):
//   out[j][c] = a1(c) sum_k M1[k][j] X1[k][c] + a2 sum_k M2[k][j] X2[k][c]
//   a1(c) = a1_kx0 for c < kx0_cols, else a1_rest
// CTA tile: TJ rows j x 64 columns c, all k; one warp per 32 x 32.  TJ is 32
// up to 32 states, else 64 (row tiles of 64 beyond).  A tile's load, product
// and epilogue follow one another, so it takes several small blocks per SM to
// keep the FP64 tensor pipe busy through the others' epilogues.  Measured
// against 128-row tiles of eight warps, two per SM: 32 states, 8276
// coefficients, rotation with velocity and planes 15.8 -> 8.5 us (six of eight
// warps had no rows); 56 states 40 -> 23; 128 states, 40115 coefficients 171 -> 130,
// plain 95 -> 75 (mean of the two products of a step), two-term 198 -> 184; 512
// states 4.72 -> 4.41 ms.  The M and X slabs of 16 k rows move through a cp.async
// ring; the two terms run as one slab sequence.  The first term's sum is
// scaled by a1(c) in registers once it is complete; the second term's M
// fragments are scaled by a2 as they are read, so one accumulator set serves
// both terms.
// ---------------------------------------------------------------------------
#define DB_TC 64
#define DB_KS 16
#define DB_LDX (DB_TC + 4)
template <int TJ> struct DbTile {
  static constexpr int THREADS = TJ * 2;
  static constexpr int BLOCKS = 256 / TJ;  // resident per SM
  static constexpr int STAGES = 3;
  static constexpr int LDM = TJ + 4;
  static constexpr int MSLAB = DB_KS * LDM, XSLAB = DB_KS * DB_LDX;
  static constexpr size_t SMEM = (size_t)STAGES * (MSLAB + XSLAB) * sizeof(double);
};

template <int TJ>
__device__ __forceinline__ void db_load_slab(double* ms, double* xs, const double* __restrict__ M,
                                             const double* __restrict__ X, int nj, int nk, long ncol, int k0,
                                             long c0, int j0) {
  typedef DbTile<TJ> D;
  if (nj & 1) {
    // odd nj: the rows of M are not 16-byte aligned; 8-byte pieces, 8 per thread
#pragma unroll
    for (int q = 0; q < (DB_KS * TJ) / D::THREADS; ++q) {
      const int piece = threadIdx.x + q * D::THREADS;
      const int kk = piece / TJ, jj = piece % TJ;
      const int k = k0 + kk;
      const bool valid = (k < nk) && (j0 + jj < nj);
      dg_cp8(ms + kk * D::LDM + jj, valid ? M + (size_t)k * nj + j0 + jj : M, valid);
    }
  } else {
    // M rows k0..k0+15, all TJ j: pieces of 16 B, 4 per thread
#pragma unroll
    for (int q = 0; q < (DB_KS * TJ / 2) / D::THREADS; ++q) {
      const int piece = threadIdx.x + q * D::THREADS;
      const int kk = piece / (TJ / 2), jj = piece % (TJ / 2) * 2;
      const int k = k0 + kk;
      const bool valid = (k < nk) && (j0 + jj < nj);
      dg_cp16(ms + kk * D::LDM + jj, valid ? M + (size_t)k * nj + j0 + jj : M, valid);
    }
  }
  // X rows k0..k0+15, columns c0..c0+63: 16 x 32 pieces
#pragma unroll
  for (int q = 0; q < (DB_KS * DB_TC / 2) / D::THREADS; ++q) {
    const int piece = threadIdx.x + q * D::THREADS;
    const int kk = piece >> 5, cc = (piece & 31) * 2;
    const int k = k0 + kk;
    const long c = c0 + cc;
    const bool valid = (k < nk) && (c < ncol);
    dg_cp16(xs + kk * DB_LDX + cc, valid ? X + (size_t)k * ncol + c : X, valid);
  }
}

// Epilogue options: yadd (optional) adds yadd[j][c] to the result (it may
// be the output array itself: each element is read and written by one
// thread); out2 (optional) receives a second copy of the result when
// *cond2 != 0; vel (optional, when *vcond != 0) receives the finite
// difference (result - previous out) vscale, previous out read by the
// thread that overwrites it.
// EDGE: the lower 32 rows of the last row tile hold no state
template <int TJ, bool TWO, bool EDGE>
__global__ void __launch_bounds__(DbTile<TJ>::THREADS, DbTile<TJ>::BLOCKS)
k_dgemm_bwd(const double* __restrict__ M1, const double* __restrict__ X1, double a1_kx0, double a1_rest,
            const double* __restrict__ M2, const double* __restrict__ X2, double a2, int nj, int nk, long ncol,
            long kx0_cols, double* out, const int* __restrict__ cond, const double* yadd, double* __restrict__ out2,
            const int* __restrict__ cond2, OaPlaneOut po, double* __restrict__ vel, double vscale,
            const int* __restrict__ vcond) {
  if (cond && *cond == 0) return;
  const bool dual = out2 && *cond2 != 0;
  const bool velo = vel && *vcond != 0;
  typedef DbTile<TJ> D;
  extern __shared__ __align__(16) double db_smem[];
  double* Ms = db_smem;
  double* Xs = db_smem + D::STAGES * D::MSLAB;
  const long c0 = (long)blockIdx.x * DB_TC;
  const int j0 = blockIdx.y * TJ;  // first row of the output tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the row block of a warp pair rotates with the block: the idle blocks of
  // an edge tile then fall on different SM sub-partitions in neighbouring
  // blocks
  const int wj = (((warp >> 1) + (EDGE ? (blockIdx.x & 1) : 0)) & (TJ / 32 - 1)) * 32, wc = (warp & 1) * 32;
  const bool live = !EDGE || j0 + wj < nj;
  const int nsl = (nk + DB_KS - 1) / DB_KS;
  const int ntot = TWO ? 2 * nsl : nsl;
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) { acc[a][b][0] = 0.0; acc[a][b][1] = 0.0; }
  auto issue = [&](int s) {
    const int st = s % D::STAGES;
    const bool second = TWO && s >= nsl;
    const int k0 = (second ? s - nsl : s) * DB_KS;
    db_load_slab<TJ>(Ms + st * D::MSLAB, Xs + st * D::XSLAB, second ? M2 : M1, second ? X2 : X1, nj, nk, ncol, k0, c0,
                 j0);
  };
  // a1(c) for this thread's output columns
  auto scale_a1 = [&]() {
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const long c = c0 + wc + b * 8 + 2 * (lane & 3) + e;
        const double a1 = (c < kx0_cols) ? a1_kx0 : a1_rest;
#pragma unroll
        for (int a = 0; a < 4; ++a) acc[a][b][e] *= a1;
      }
  };
#pragma unroll
  for (int s = 0; s < D::STAGES - 1; ++s) {
    if (s < ntot) issue(s);
    dg_commit();
  }
  for (int s = 0; s < ntot; ++s) {
    dg_wait<D::STAGES - 2>();
    __syncthreads();
    if (s + D::STAGES - 1 < ntot) issue(s + D::STAGES - 1);
    dg_commit();
    if (TWO && s == nsl) scale_a1();
    const double sa = (TWO && s >= nsl) ? a2 : 1.0;
    const double* ms = Ms + (s % D::STAGES) * D::MSLAB;
    const double* xs = Xs + (s % D::STAGES) * D::XSLAB;
    if (live)
#pragma unroll
    for (int k4 = 0; k4 < DB_KS; k4 += 4) {
      double af[4], bf[4];
      // A[j][k] = M[k][j] (row-major 8 x 4 fragment), B[k][c] = X[k][c]
#pragma unroll
      for (int q = 0; q < 4; ++q) af[q] = ms[(k4 + (lane & 3)) * D::LDM + wj + q * 8 + (lane >> 2)] * sa;
#pragma unroll
      for (int q = 0; q < 4; ++q) bf[q] = xs[(k4 + (lane & 3)) * DB_LDX + wc + q * 8 + (lane >> 2)];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) dg_dmma(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
    }
  }
  dg_wait<0>();
  if (!TWO) scale_a1();
  // the old out or yadd (which may be out) of eight pieces is read before any
  // of them is written: read one at a time behind the writes they were a
  // chain of sixteen L2 round trips, 8 of 13 us at 32 states
  const double* pre = velo ? out : yadd;
#pragma unroll
  for (int a2 = 0; a2 < 4; a2 += 2) {
    double2 p[2][4];
    if (pre) {
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int j = j0 + wj + (a2 + a) * 8 + (lane >> 2);
          const long c = c0 + wc + b * 8 + 2 * (lane & 3);
          p[a][b] = make_double2(0.0, 0.0);
          if (j < nj && c < ncol) p[a][b] = *(const double2*)(pre + (size_t)j * ncol + c);
        }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int j = j0 + wj + (a2 + a) * 8 + (lane >> 2);
      if (j >= nj) continue;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const long c = c0 + wc + b * 8 + 2 * (lane & 3);  // even, as ncol is
        const size_t o = (size_t)j * ncol + c;
        if (c >= ncol) continue;
        double2 v = make_double2(acc[a2 + a][b][0], acc[a2 + a][b][1]);
        if (velo) {
          *(double2*)(vel + o) = make_double2(fma(v.x, vscale, p[a][b].x * -vscale), fma(v.y, vscale, p[a][b].y * -vscale));
        } else if (pre) {
          v.x += p[a][b].x;
          v.y += p[a][b].y;
        }
        *(double2*)(out + o) = v;
        if (dual) *(double2*)(out2 + o) = v;
      }
    }
  }
  if (po.P) {
    // bf16 planes of the tile staged in the (now idle) slab ring, then
    // written as whole 16-byte pieces of 128-byte rows
    constexpr int SPLD = DB_TC + 8;
    __nv_bfloat16* sp = reinterpret_cast<__nv_bfloat16*>(db_smem);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int jl = wj + a * 8 + (lane >> 2);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int cl = wc + b * 8 + 2 * (lane & 3);
        __nv_bfloat162 h[3];
        oa_bf16_digits2(acc[a][b][0], acc[a][b][1], po.nt, h);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (q >= po.nt) break;
          *reinterpret_cast<__nv_bfloat162*>(sp + ((size_t)q * TJ + jl) * SPLD + cl) = h[q];
        }
      }
    }
    __syncthreads();
    const size_t pstride = (size_t)po.rows_pad * po.ldp;
    for (int i = threadIdx.x; i < po.nt * TJ * (DB_TC / 8); i += D::THREADS) {
      const int q = i / (TJ * (DB_TC / 8)), rem = i - q * (TJ * (DB_TC / 8));
      const int jl = rem / (DB_TC / 8), ch = rem - jl * (DB_TC / 8);
      if (j0 + jl >= nj || c0 + ch * 8 >= po.ldp) continue;
      *reinterpret_cast<uint4*>((__nv_bfloat16*)po.P + q * pstride +
                                oa_plane_at(j0 + jl, c0 + ch * 8, po.rows_pad)) =
          *reinterpret_cast<const uint4*>(sp + ((size_t)q * TJ + jl) * SPLD + ch * 8);
    }
  }
}

// Returns cudaErrorNotSupported when the shapes or pointers do not allow the
// copies (odd ncol, unaligned pointers); an odd nj moves M in 8-byte pieces.
// Outputs of more than 64 rows run as row tiles of 64 (grid y).
// po (optional): bf16 planes of out written in the same pass (ncol even).
cudaError_t oa_dgemm_bwd_ex(cudaStream_t s, const double* M1, const double* X1, double a1_kx0, double a1_rest,
                            const double* M2, const double* X2, double a2, int nj, int nk, long ncol, long kx0_cols,
                            double* out, const int* cond, const double* yadd, double* out2, const int* cond2,
                            const OaPlaneOut* po, double* vel, double vscale, const int* vcond) {
  const OaPlaneOut pz = po ? *po : OaPlaneOut{nullptr, 0, 0, 0};
  if (vel && (!vcond || yadd || M2)) return cudaErrorInvalidValue;
  // plane tiles are whole 64-column pieces inside the plane rows
  if (pz.P && ((pz.ldp % DB_TC) || ncol > pz.ldp || nj > pz.rows_pad || pz.nt > 3)) return cudaErrorInvalidValue;
  const uintptr_t al = (uintptr_t)M1 | (uintptr_t)X1 | (uintptr_t)out | (uintptr_t)(M2 ? M2 : M1) |
                       (uintptr_t)(X2 ? X2 : X1) | (uintptr_t)yadd | (uintptr_t)out2 | (uintptr_t)vel;
  if (out2 && !cond2) return cudaErrorInvalidValue;
  if (nj <= 0 || (ncol & 1) || (al & 15) || nk <= 0 || (M2 && !X2)) return cudaErrorNotSupported;
  // column tiles of 64 by row tiles of tj
  auto go = [&](auto kern, int tj, int threads, size_t sm) -> cudaError_t {
    const cudaError_t e = oa_smem_limit(kern);
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((ncol + DB_TC - 1) / DB_TC), (unsigned)((nj + tj - 1) / tj));
    kern<<<grid, threads, sm, s>>>(M1, X1, a1_kx0, a1_rest, M2, X2, a2, nj, nk, ncol, kx0_cols, out, cond, yadd, out2,
                                   cond2, pz, vel, vscale, vcond);
    return cudaGetLastError();
  };
#define OA_DB(TJ, EDGE)                                                                             \
  return M2 ? go(k_dgemm_bwd<TJ, true, EDGE>, TJ, DbTile<TJ>::THREADS, DbTile<TJ>::SMEM)            \
            : go(k_dgemm_bwd<TJ, false, EDGE>, TJ, DbTile<TJ>::THREADS, DbTile<TJ>::SMEM)
  if (nj <= 32) OA_DB(32, false);
  if (nj % 64 >= 1 && nj % 64 <= 32) OA_DB(64, true);
  OA_DB(64, false);
#undef OA_DB
}

cudaError_t oa_dgemm_bwd(cudaStream_t s, const double* M1, const double* X1, double a1_kx0, double a1_rest,
                         const double* M2, const double* X2, double a2, int nj, int nk, long ncol, long kx0_cols,
                         double* out, const int* cond) {
  return oa_dgemm_bwd_ex(s, M1, X1, a1_kx0, a1_rest, M2, X2, a2, nj, nk, ncol, kx0_cols, out, cond, nullptr, nullptr,
                         nullptr, nullptr, nullptr, 0.0, nullptr);
}
