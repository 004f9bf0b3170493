// EES nonlocal path on state pairs (oa_pp.cuh's transform on the nonlocal
// grid, nx = ny = N):
//   k_pe_gather   z-line rows of a pair -> y FFT -> x FFT -> Z partials (and
//                 atom-force sums) of the atoms whose stencils meet plane z
//   k_pe_scatter  zs of a pair on the stencils -> x^-1 -> y^-1 -> z-line rows
// A plane meets only natm order / nc stencils (five or six atoms of 128 on a
// 96 grid), so only the rows that those stencils touch (about 20 of 96) are
// transformed along x: the gather takes no other row from the y transform,
// and the scatter hands zeros for the others to it.  The x transform of a row
// stays in its warp: its values go through the warp's slice of shared memory
// to the stencil sums, with no tile of the whole plane.
//
// Measured at 128 waters (512 states, 96^3, FP32) against the per-state plane
// kernels: gather 2.20 -> 0.64 ms, scatter 2.08 -> 0.71 ms (beside the density
// path); 60^3, FP64, 120 states: 181 and 131 us.
//
// Reference work replaced: eesZmatRchare / eesEnergyAtmForcRchare on the
// nonlocal grid (cp_ees_nonlocal.C:1238-1352, 1480-1720) with the plane
// transforms of fftCache.C:562-816.
#pragma once
#include "oa_pp.cuh"

// strides as PpCfg; W warps, RG rows per warp at a time, MB resident blocks
template <typename R_, int N1_, int N2_, int LSX_, int PS_, int LSP_, int LDM_, int W_, int RG_, int MB_>
struct PeCfg {
  typedef R_ R;
  typedef typename CplxOf<R_>::T C;
  static constexpr int N1 = N1_, N2 = N2_, N = N1_ * N2_;
  static constexpr int LSX = LSX_, PS = PS_, LSP = LSP_;
  static constexpr int LDP = pp_stride(N1_ * LSP_, LDM_, 128 / (int)sizeof(C));
  static constexpr int TP = N1_ | 1, RW = 32 / N2_, RWI = RW * N2_;
  static constexpr int W = W_, RG = RG_, MB = MB_;
  static constexpr int NS = N | 1;  // natural-order row of x values
  template <bool BAND> static __host__ __device__ constexpr bool dead(int) { return false; }
};

struct PeSmem {
  size_t T, col, rows, P, S, ent, tot;
  int lr;
};

// Per block: the rows of plane z that stencils touch (mask[k1] bit k2 for row
// y = k1 + N1 k2, list of them) and the stencil rows on each: entries
// [first[r], first[r + 1]) of ent, (atom << 8) | (b index << 4) | c index, in
// atom order.  One warp builds them.
template <int N1, int N2>
__device__ __forceinline__ void pe_plane_rows(const EesArgs& E, int z, int* ent, unsigned* mask, int* list,
                                              int* first, int* count) {
  constexpr int N = N1 * N2;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    for (int k = lane; k < N1; k += 32) mask[k] = 0u;
    for (int k = lane; k <= N; k += 32) first[k] = 0;
    __syncwarp();
    // c index of an atom's stencil on this plane, -1: none
    auto on_plane = [&](int a) {
      const int* ic = E.idx + ((size_t)a * 3 + 2) * E.order;
      int jc = -1;
      for (int j = 0; j < E.order; ++j)
        if (ic[j] == z) jc = j;
      return jc;
    };
    for (int a = lane; a < E.natm; a += 32)
      if (on_plane(a) >= 0) {
        const int* ib = E.idx + ((size_t)a * 3 + 1) * E.order;
        for (int j = 0; j < E.order; ++j) {
          atomicOr(&mask[ib[j] % N1], 1u << (ib[j] / N1));
          atomicAdd(&first[ib[j] + 1], 1);  // entries per row y, shifted by one
        }
      }
    __syncwarp();
    if (lane == 0) {
      int nr = 0, sum = 0;
      for (int y = 0; y < N; ++y) {
        const int c = first[y + 1];
        if (c > 0) {
          list[nr] = y;
          first[nr] = sum;
          ++nr;
          sum += c;
        }
      }
      first[nr] = sum;
      count[0] = nr;
    }
    __syncwarp();
    const int nr = count[0];
    for (int r = lane; r < nr; r += 32) {
      int o = first[r];
      for (int a = 0; a < E.natm && o < first[r + 1]; ++a) {
        const int jc = on_plane(a);
        if (jc < 0) continue;
        const int* ib = E.idx + ((size_t)a * 3 + 1) * E.order;
        for (int j = 0; j < E.order; ++j)
          if (ib[j] == list[r]) ent[o++] = (a << 8) | (j << 4) | jc;
      }
    }
  }
}

template <class F>
__global__ void __launch_bounds__(F::W * 32, F::MB)
k_pe_gather(const typename F::C* __restrict__ zbuf, int nstate, int nz, int ldl, const int4* __restrict__ cols,
            int nkx, const double2* __restrict__ twg, int ngroup, EesArgs E, PeSmem L) {
  typedef typename F::C C;
  typedef typename F::R R;
  constexpr int N1 = F::N1, N2 = F::N2, N = F::N, LDP = F::LDP, LSP = F::LSP, LSX = F::LSX, PS = F::PS, NS = F::NS;
  constexpr int W = F::W, RG = F::RG, RW = F::RW, EPC = 16 / (int)sizeof(C);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned mask[N1];
  __shared__ int list[N], first[N + 1], count[1];
  C* T = (C*)(smem_raw + L.T);
  int4* col = (int4*)(smem_raw + L.col);
  C* rows = (C*)(smem_raw + L.rows);
  C* P = (C*)(smem_raw + L.P);
  int* ent = (int*)(smem_raw + L.ent);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int la = lane / N2, n2 = lane - la * N2;
  C* Sx = (C*)(smem_raw + L.S) + wid * (RG * (PS > NS ? PS : NS));
  const int z = blockIdx.x, g = blockIdx.y;
  const int npair = (nstate + 1) / 2;
  const int qb = (int)((long)g * npair / ngroup), qe = (int)((long)(g + 1) * npair / ngroup);
  const int ncol = 2 * nkx - 1, cpw = (ncol + W - 1) / W, c0 = min(wid * cpw, ncol), ncw = min(cpw, ncol - c0);
  const bool frc = E.fpart != nullptr;
  pp_load_tw<F>(T, twg);
  for (int i = threadIdx.x; i < nkx; i += W * 32) col[i] = cols[i];
  pe_plane_rows<N1, N2>(E, z, ent, mask, list, first, count);
  __syncthreads();
  const int nrow = count[0];
  if (nrow == 0) return;  // no stencil meets this plane
  const int rpw = (nrow + W - 1) / W, rw0 = min(wid * rpw, nrow), nrw = min(rpw, nrow - rw0);
  auto stage = [&](int q) {
    if (L.lr) {
      const int nch = L.lr / EPC;
      for (int i = threadIdx.x; i < 2 * nch; i += W * 32) {
        const int st = i >= nch ? 1 : 0, ch = i - st * nch;
        const int s = 2 * q + st;
        if (s < nstate) pp_cp16(rows + st * L.lr + EPC * ch, zbuf + ((size_t)s * nz + z) * ldl + EPC * ch);
      }
      asm volatile("cp.async.commit_group;\n" ::);
    }
  };
  if (qb < qe) stage(qb);
  const PpTw<F, sizeof(R) == 4> tw(T, n2);
  for (int q = qb; q < qe; ++q) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    {
      const bool has1 = 2 * q + 1 < nstate;
      const C* rA = L.lr ? rows : zbuf + ((size_t)(2 * q) * nz + z) * ldl;
      const C* rB = L.lr ? rows + L.lr : rA + (size_t)nz * ldl;
      for (int c = la; la < RW && c < ncw; c += RW) {
        const int kx = c0 + c - (nkx - 1);
        C u[N1];
        pp_load_col<F, false>(u, rA, rB, has1, col[kx < 0 ? -kx : kx], kx, n2);
        RDft<N1, -1>::run(u);
        C* p = P + (c0 + c) * LDP + n2;
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) p[k1 * LSP] = k1 ? tw.template mul<-1>(u[k1], k1) : u[0];
      }
      __syncwarp();
      for (int it = lane; it < ncw * N1; it += 32) {
        const int c = it / N1, k1 = it - c * N1;
        if (mask[k1] == 0u) continue;
        C* p = P + (c0 + c) * LDP + k1 * LSP;
        C w[N2];
#pragma unroll
        for (int i = 0; i < N2; ++i) w[i] = p[i];
        RDft<N2, -1>::run(w);
#pragma unroll
        for (int i = 0; i < N2; ++i) p[i] = w[i];
      }
    }
    __syncthreads();
    if (q + 1 < qe) stage(q + 1);
    for (int r0 = 0; r0 < nrw; r0 += RG) {
      const int nr = min(RG, nrw - r0);
#pragma unroll
      for (int j = 0; j < pp_ceil(RG, RW); ++j) {
        const int rr = la + RW * j;
        if (la < RW && rr < nr) {
          const int y = list[rw0 + r0 + rr], rk = y % N1;
          const C* p = P + rk * LSP + y / N1;
          C u[N1];
#pragma unroll
          for (int n1 = 0; n1 < N1; ++n1) {
            const int k = N2 * n1 + n2;
            const int kx = 2 * k <= N ? k : k - N;
            u[n1] = cmk<C>(0.0, 0.0);
            if (kx < nkx && -kx < nkx) u[n1] = p[(kx + nkx - 1) * LDP];
          }
          RDft<N1, -1>::run(u);
          C* sx = Sx + rr * PS + n2;
          sx[0] = u[0];
#pragma unroll
          for (int k1 = 1; k1 < N1; ++k1) sx[k1 * LSX] = tw.template mul<-1>(u[k1], k1);
        }
      }
      __syncwarp();
      // x pass B: the rows' values replace the pass-A buffer in natural order
      constexpr int XB = pp_ceil(RG * N1, 32);
      C w[XB][N2];
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        const int it = lane + 32 * j;
        const int rr = it / N1, k1 = it - rr * N1;
        if (rr < nr) {
#pragma unroll
          for (int i = 0; i < N2; ++i) w[j][i] = Sx[rr * PS + k1 * LSX + i];
          RDft<N2, -1>::run(w[j]);
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        const int it = lane + 32 * j;
        const int rr = it / N1, k1 = it - rr * N1;
        if (rr < nr) {
#pragma unroll
          for (int i = 0; i < N2; ++i) Sx[rr * NS + k1 + N1 * i] = w[j][i];
        }
      }
      __syncwarp();
      // row sums of the stencils, lanes over the entries of these rows:
      // zpart[s][a][c index][b index] = M_c M_b sum_ja psi M_a
      const int e0 = first[rw0 + r0], e1 = first[rw0 + r0 + nr];
      for (int e = e0 + lane; e < e1; e += 32) {
        int rr = 0;
        while (rr + 1 < nr && e >= first[rw0 + r0 + rr + 1]) ++rr;
        const int a = ent[e] >> 8, jb = (ent[e] >> 4) & 15, jc = ent[e] & 15;
        const int* ix = E.idx + (size_t)a * 3 * E.order;
        const double* m = E.mn + (size_t)a * 3 * E.order;
        const double* d = frc ? E.dmn + (size_t)a * 3 * E.order : m;
        double sa = 0.0, sb = 0.0, da = 0.0, db = 0.0;
        for (int ja = 0; ja < E.order; ++ja) {
          const C v = Sx[rr * NS + ix[ja]];
          sa += (double)v.x * m[ja];
          sb += (double)v.y * m[ja];
          if (frc) {
            da += (double)v.x * d[ja];
            db += (double)v.y * d[ja];
          }
        }
        const double mb = m[E.order + jb], mc = m[2 * E.order + jc];
        const size_t o = (((size_t)(2 * q) * E.natm + a) * E.order + jc) * E.order + jb;
        const size_t o2 = o + (size_t)E.natm * E.order * E.order;
        const bool has1 = 2 * q + 1 < nstate;
        E.zpart[o] = sa * mb * mc;
        if (has1) E.zpart[o2] = sb * mb * mc;
        if (frc) {
          const double eb = d[E.order + jb], ec = d[2 * E.order + jc];
          double* f = E.fpart + 3 * o;
          f[0] = da * mb * mc; f[1] = sa * eb * mc; f[2] = sa * mb * ec;
          if (has1) {
            f = E.fpart + 3 * o2;
            f[0] = db * mb * mc; f[1] = sb * eb * mc; f[2] = sb * mb * ec;
          }
        }
      }
      __syncwarp();
    }
  }
}

template <class F>
__global__ void __launch_bounds__(F::W * 32, F::MB)
k_pe_scatter(typename F::C* __restrict__ zbuf, int nstate, int nz, int ldl, int nlines, const int4* __restrict__ cols,
             int nkx, const double2* __restrict__ twg, int ngroup, EesArgs E, PeSmem L) {
  typedef typename F::C C;
  typedef typename F::R R;
  constexpr int N1 = F::N1, N2 = F::N2, N = F::N, LDP = F::LDP, LSP = F::LSP, LSX = F::LSX, PS = F::PS, NS = F::NS;
  constexpr int W = F::W, RG = F::RG, RW = F::RW, XB = pp_ceil(RG * N1, 32);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned mask[N1];
  __shared__ int list[N], first[N + 1], count[1];
  C* T = (C*)(smem_raw + L.T);
  int4* col = (int4*)(smem_raw + L.col);
  C* P = (C*)(smem_raw + L.P);
  int* ent = (int*)(smem_raw + L.ent);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int la = lane / N2, m2 = lane - la * N2;
  C* Sx = (C*)(smem_raw + L.S) + wid * (RG * (PS > NS ? PS : NS));
  const int z = blockIdx.x, g = blockIdx.y;
  const int npair = (nstate + 1) / 2;
  const int qb = (int)((long)g * npair / ngroup), qe = (int)((long)(g + 1) * npair / ngroup);
  const int kpw = (nkx + W - 1) / W, x0 = min(wid * kpw, nkx), nkw = min(kpw, nkx - x0);
  pp_load_tw<F>(T, twg);
  for (int i = threadIdx.x; i < nkx; i += W * 32) col[i] = cols[i];
  pe_plane_rows<N1, N2>(E, z, ent, mask, list, first, count);
  __syncthreads();
  const int nrow = count[0];
  if (nrow == 0) {
    // no stencil meets this plane: its rows are zero
    for (int q = qb; q < qe; ++q)
      for (int st = 0; st < 2; ++st)
        if (2 * q + st < nstate)
          for (int l = threadIdx.x; l < nlines; l += W * 32)
            zbuf[((size_t)(2 * q + st) * nz + z) * ldl + l] = cmk<C>(0.0, 0.0);
    return;
  }
  const int rpw = (nrow + W - 1) / W, rw0 = min(wid * rpw, nrow), nrw = min(rpw, nrow - rw0);
  const PpTw<F, sizeof(R) == 4> tw(T, m2);
  for (int q = qb; q < qe; ++q) {
    const bool has1 = 2 * q + 1 < nstate;
    const double* za = E.zs + (size_t)(2 * q) * E.natm;
    const double* zb = za + E.natm;
    for (int r0 = 0; r0 < nrw; r0 += RG) {
      const int nr = min(RG, nrw - r0);
      for (int i = lane; i < nr * NS; i += 32) Sx[i] = cmk<C>(0.0, 0.0);
      __syncwarp();
      // z M_a M_b M_c of every stencil row, one after the other, lanes over
      // the a index
      for (int rr = 0; rr < nr; ++rr)
        for (int e = first[rw0 + r0 + rr]; e < first[rw0 + r0 + rr + 1]; ++e) {
          const int a = ent[e] >> 8, jb = (ent[e] >> 4) & 15, jc = ent[e] & 15;
          if (lane < E.order) {
            const int* ix = E.idx + (size_t)a * 3 * E.order;
            const double* m = E.mn + (size_t)a * 3 * E.order;
            const double mm = m[2 * E.order + jc] * m[E.order + jb] * m[lane];
            C& v = Sx[rr * NS + ix[lane]];
            v.x += (R)(za[a] * mm);
            if (has1) v.y += (R)(zb[a] * mm);
          }
          __syncwarp();
        }
      C w[XB][N2];
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        const int it = lane + 32 * j;
        const int rr = it / N1, k1 = it - rr * N1;
        if (rr < nr) {
#pragma unroll
          for (int i = 0; i < N2; ++i) w[j][i] = Sx[rr * NS + k1 + N1 * i];
          RDft<N2, +1>::run(w[j]);
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        const int it = lane + 32 * j;
        const int rr = it / N1, k1 = it - rr * N1;
        if (rr < nr) {
#pragma unroll
          for (int i = 0; i < N2; ++i) Sx[rr * PS + k1 * LSX + i] = w[j][i];
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < pp_ceil(RG, RW); ++j) {
        const int rr = la + RW * j;
        if (la < RW && rr < nr) {
          C u[N1];
          const C* sx = Sx + rr * PS + m2;
          u[0] = sx[0];
#pragma unroll
          for (int k1 = 1; k1 < N1; ++k1) u[k1] = tw.template mul<+1>(sx[k1 * LSX], k1);
          RDft<N1, +1>::run(u);
          const int y = list[rw0 + r0 + rr], rk = y % N1;
          C* p = P + rk * LSP + y / N1;
#pragma unroll
          for (int m1 = 0; m1 < N1; ++m1) {
            const int k = m2 + N2 * m1;
            const int kx = 2 * k <= N ? k : k - N;
            if (kx < nkx && -kx < nkx) p[(kx + nkx - 1) * LDP] = u[m1];
          }
        }
      }
      __syncwarp();
    }
    __syncthreads();
    // y phase: rows outside the list are zero
    for (int it = lane; it < 2 * nkw * N1; it += 32) {
      const int c = it / N1, k1 = it - c * N1;
      const int ax = x0 + (c >> 1);
      const bool neg = c & 1;
      if (neg && ax == 0) continue;
      C* p = P + (nkx - 1 + (neg ? -ax : ax)) * LDP + k1 * LSP;
      const unsigned mk = mask[k1];
      C w[N2];
#pragma unroll
      for (int i = 0; i < N2; ++i) {
        w[i] = cmk<C>(0.0, 0.0);
        if (mk >> i & 1u) w[i] = p[i];
      }
      if (mk) RDft<N2, +1>::run(w);
#pragma unroll
      for (int i = 0; i < N2; ++i) p[i] = w[i];
    }
    __syncwarp();
    pp_store_cols<F, false, true>(zbuf + ((size_t)(2 * q) * nz + z) * ldl, (size_t)nz * ldl, has1, P, LDP, col, nkx, x0,
                            nkw, lane, T, tw);
    __syncthreads();
  }
}

// shared-memory layout; tot = 0 when it does not fit
template <class F>
static PeSmem pe_layout(int mode, int nkx, int nlines, int natm, int order) {
  typedef typename F::C C;
  constexpr int EPC = 16 / (int)sizeof(C);
  auto make = [&](bool staged) {
    PeSmem L;
    size_t o = 0;
    L.lr = staged ? (nlines + EPC - 1) / EPC * EPC : 0;
    L.T = o; o += align_up((size_t)F::N2 * F::TP * sizeof(C), 16);
    L.col = o; o += align_up((size_t)nkx * sizeof(int4), 16);
    L.rows = o; o += align_up((size_t)2 * L.lr * sizeof(C), 16);
    L.P = o; o += align_up((size_t)(2 * nkx - 1) * F::LDP * sizeof(C), 16);
    L.S = o; o += align_up((size_t)F::W * F::RG * (F::PS > F::NS ? F::PS : F::NS) * sizeof(C), 16);
    L.ent = o; o += align_up((size_t)natm * order * sizeof(int), 16);
    L.tot = o;
    return L;
  };
  const size_t lim = (size_t)OA_MAX_SMEM - 2048;  // static shared memory of the kernels
  PeSmem L = make(mode == 2);
  if (L.tot > lim && mode == 2) L = make(false);
  if (L.tot > lim) L.tot = 0;
  return L;
}

template <class F>
static cudaError_t pe_run(const PeArgs& A) {
  typedef typename F::C C;
  if (2 * (A.nkx - 1) >= F::N || 2 * A.kymax >= F::N || (A.ldl & 1) || A.E->order > 16 || A.E->natm >= 1 << 23) return cudaErrorNotSupported;
  const PeSmem L2 = pe_layout<F>(2, A.nkx, A.nlines, A.E->natm, A.E->order);
  const PeSmem L3 = pe_layout<F>(3, A.nkx, A.nlines, A.E->natm, A.E->order);
  if (!L2.tot || !L3.tot) return cudaErrorNotSupported;
  if (A.mode < 0) {
    cudaError_t e = oa_smem_limit(k_pe_gather<F>);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(A.bps, k_pe_gather<F>, F::W * 32, L2.tot);
  }
  const dim3 grid(A.nz, A.ngroup);
  if (A.mode == 2) {
    cudaError_t e = oa_smem_limit(k_pe_gather<F>);
    if (e != cudaSuccess) return e;
    k_pe_gather<F><<<grid, F::W * 32, L2.tot, A.st>>>((const C*)A.zbuf, A.nstate, A.nz, A.ldl, (const int4*)A.cols,
                                                      A.nkx, A.tw, A.ngroup, *A.E, L2);
  } else {
    cudaError_t e = oa_smem_limit(k_pe_scatter<F>);
    if (e != cudaSuccess) return e;
    k_pe_scatter<F><<<grid, F::W * 32, L3.tot, A.st>>>((C*)A.zbuf, A.nstate, A.nz, A.ldl, A.nlines,
                                                       (const int4*)A.cols, A.nkx, A.tw, A.ngroup, *A.E, L3);
  }
  return cudaGetLastError();
}
