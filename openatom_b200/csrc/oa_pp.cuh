// State-pair plane kernels of the state FFT path, for every grid length with
// a two-pass factorisation N = N1 N2 (oa_rdft.cuh) and both precision forms
// (FP64 without 125, 150 and 160, whose planes do not fit):
//   k_pp_density  z-line rows -> psi(r) of two states -> density sum, psi(r) stored
//   k_pp_vks      stored psi(r) V_KS -> z-line rows
//
// Two real states share one complex plane transform: with c = psi_a + i psi_b
// the plane's spectrum is c(kx, ky) = a(kx, ky) + i b(kx, ky) for kx >= 0 and
// conj a(-kx, -ky) + i conj b(-kx, -ky) for kx < 0, so the y pass combines
// the two states' z-line runs as it loads them (2 nkx - 1 complex columns),
// everything after is a plain complex transform, and the backward kernel
// separates the states as it stores (both columns +-kx of an element pair in
// one thread's registers).  A plane pair makes four shared-memory round trips
// over half planes or planes:
//   y pass A  (thread = column, n2): DFT_N1 -> P[column][k1][n2]
//   y pass B  (thread = column, k1): DFT_N2 in place, P[column][k1][k2];
//             row y = k1 + N1 k2 sits at position k1 LSP + k2
//   x pass A  (thread = row, n2): DFT_N1 over the kx columns -> Sx[row][k1][n2]
//   x pass B  (thread = row, k1): DFT_N2 -> psi(x = k1 + N1 k2) of the pair
// and the same backwards.  Each warp owns its columns in the y phase and its
// rows in the x phase (its own Sx slice), so passes A and B of a phase are
// separated by __syncwarp only and a pair costs two block barriers.  Row to
// thread assignment is fixed, so the density of a plane (and, in FP32, V_KS)
// stays in registers over all pairs of a block.
// HS > 1 (long FP64 planes): a block takes 1 / HS of the k1 classes of the
// rows, which divides P and the register sums by HS at the price of
// repeating y pass A.
//
// psi(r) is private to the two kernels: [pair][z][k2][row position][k1], the
// order in which pass B holds it, so that stores and loads are contiguous.
//
// What bounds them: the shared-memory round trips and the instructions of the
// register DFTs (DRAM traffic is psi(r) and the z-lines once).  Measured,
// density / V_KS: 108^3, 128 states, FP32 287 / 286 us (one pair per block
// iteration with block barriers between the passes: 305 / 331), FP64 554 / 542 us
// (per-state planes: 1093 / 963); 120^3, 256 states, FP64 1.73 / 1.43 ms
// (runtime-plan planes: 15.8 together); 80^3, 78 states, FP32 50 / 56 us.
//
// Shared-memory strides are chosen per length by enumeration over the access
// patterns above (bank conflicts of 8- or 16-byte elements); the table is in
// oa_pp_table.h.
//
// Reference work replaced:
//   FFTcache::doStpFFTGtoR_Rchare (fftCache.C:1167) + the density part of
//     CP_State_RealSpacePlane::doFFT / doReduction (:349-363, 450-517)     -> k_pp_density
//   CP_State_RealSpacePlane::unpackVks (:530-597) + doStpFFTRtoG_Rchare
//     (fftCache.C:1252-1319)                                               -> k_pp_vks
#pragma once
#include "oa_rdft.cuh"
#include "oa_state_common.cuh"
#include "oa_pp.h"

__host__ __device__ constexpr int pp_ceil(int a, int b) { return (a + b - 1) / b; }
// smallest stride >= v congruent to m modulo d
__host__ __device__ constexpr int pp_stride(int v, int m, int d) { return v + ((m - v) % d + d) % d; }

// LSX, PS: x buffer [row][k1][n2]; LSP: k1 stride of P; LDM: column stride of
// P modulo the bank period; HS: row splits of the density pass; per kernel W
// warps, RG rows per warp at a time, MB resident blocks aimed for
template <typename R_, int N1_, int N2_, int LSX_, int PS_, int LSP_, int LDM_, int HS_, int WD_, int RGD_, int MBD_,
          int WV_, int RGV_, int MBV_>
struct PpCfg {
  typedef R_ R;
  typedef typename CplxOf<R_>::T C;
  static constexpr int N1 = N1_, N2 = N2_, N = N1_ * N2_;
  static constexpr int BP = 128 / (int)sizeof(C);       // elements per bank period
  static constexpr int LSX = LSX_, PS = PS_, LSP = LSP_, HS = HS_;
  static constexpr int K1H = pp_ceil(N1_, HS_);         // k1 classes of a row split
  static constexpr int RH = K1H * N2_;                  // rows of a split
  static constexpr int LDPD = pp_stride(K1H * LSP_, LDM_, BP);
  static constexpr int LDPV = pp_stride(N1_ * LSP_, LDM_, BP);
  static constexpr int TP = N1_ | 1;                    // twiddle table T[n2][k1]
  // A steps: FP32 gives each lane a fixed n2 (lane = pencil N2 + n2, RW pencils
  // at a time), so that its twiddles stay in registers for a phase (they are
  // a third of the shared-memory traffic otherwise); FP64 has no registers
  // for them and walks (pencil, n2) items with every lane busy.  At 108^3,
  // 128 states, FP32: density 299 -> 288 us, V_KS 306 -> 285 us; FP64 the
  // other way round: density 529 -> 594 us, V_KS 512 -> 615 us with fixed lanes.
  static constexpr bool FIX = sizeof(R_) == 4;
  static constexpr int RW = 32 / N2_;
  static constexpr int RWI = FIX ? RW * N2_ : 32;       // items of a warp per A step
  static constexpr int WD = WD_, RGD = RGD_, MBD = MBD_;
  static constexpr int RPD = pp_ceil(RH, WD_), NGD = pp_ceil(RPD, RGD_);
  static constexpr int WV = WV_, RGV = RGV_, MBV = MBV_;
  static constexpr int RPV = pp_ceil(N, WV_), NGV = pp_ceil(RPV, RGV_);
  static constexpr bool CANBAND = N1_ % 4 == 0;
  // DFT_N1 inputs / outputs that lie outside a band |k| < N/4
  template <bool BAND> static __host__ __device__ constexpr bool dead(int n1) {
    return BAND && n1 >= N1_ / 4 && n1 < 3 * N1_ / 4;
  }
};

struct PpSmem {
  size_t T, col, rows, P, S, total;
  int lr;  // staged z-line row length in elements (0: the rows are read from global memory)
};

static __device__ __forceinline__ void pp_cp16(void* sdst, const void* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc));
}

// T[n2][k1] = exp(-2 pi i n2 k1 / N)
template <class F>
__device__ __forceinline__ void pp_load_tw(typename F::C* T, const double2* __restrict__ twg) {
  for (int i = threadIdx.x; i < F::N; i += blockDim.x) {
    const int n2 = i / F::N1, k1 = i - n2 * F::N1;
    const double2 t = twg[n2 * k1];
    T[n2 * F::TP + k1] = cmk<typename F::C>(t.x, t.y);
  }
}

// this lane's twiddles, in registers for a phase (REG) or read from the table
// at each use
template <class F, bool REG> struct PpTw {
  const typename F::C* row;
  typename F::C t[REG ? F::N1 : 1];
  __device__ __forceinline__ PpTw(const typename F::C* T, int n2) : row(T + n2 * F::TP) {
    if constexpr (REG) {
#pragma unroll
      for (int k1 = 1; k1 < F::N1; ++k1) t[k1] = row[k1];
    }
  }
  template <int SIGN> __device__ __forceinline__ typename F::C mul(typename F::C a, int k1) const {
    typename F::C w;
    if constexpr (REG) w = t[k1];
    else w = row[k1];
    if (SIGN > 0) w.y = -w.y;
    return cmul(a, w);
  }
};

// a exp(+2 pi i n2 k1 / N)
template <class F>
__device__ __forceinline__ typename F::C pp_tw_inv(typename F::C a, const typename F::C* T, int n2, int k1) {
  typename F::C w = T[n2 * F::TP + k1];
  w.y = -w.y;
  return cmul(a, w);
}

// the twiddles of an item: the lane's own (FIX) or the table row of its n2
template <class F>
__device__ __forceinline__ const PpTw<F, true>& pp_tw(const PpTw<F, true>& lane_tw, const typename F::C*, int) {
  return lane_tw;
}
template <class F>
__device__ __forceinline__ PpTw<F, false> pp_tw(const PpTw<F, false>&, const typename F::C* T, int n2) {
  return PpTw<F, false>(T, n2);
}

// DFT_N1 inputs of class n2 of column kx of the pair's spectrum c = a + i b
// (see the top of this file) from the z-line runs of the two states
template <class F, bool BAND>
__device__ __forceinline__ void pp_load_col(typename F::C* u, const typename F::C* rA, const typename F::C* rB,
                                            bool has1, int4 cr, int kx, int n2) {
  typedef typename F::C C;
  typedef typename F::R R;
  const C* a = rA + cr.x;
  const C* b = rB + cr.x;
#pragma unroll
  for (int n1 = 0; n1 < F::N1; ++n1) {
    C v = cmk<C>(0.0, 0.0);
    if (!F::template dead<BAND>(n1)) {
      const int i = F::N2 * n1 + n2;
      const int ky = 2 * i <= F::N ? i : i - F::N;
      const int l = (kx < 0 ? -ky : ky) - cr.y;
      if (l >= 0 && l < cr.z) {
        const C av = a[l];
        C bv = cmk<C>(0.0, 0.0);
        if (has1) bv = b[l];
        if (kx >= 0) { v.x = av.x - bv.y; v.y = av.y + bv.x; }
        else { v.x = av.x + bv.y; v.y = bv.x - av.y; }
      }
      if (kx == 0) {
        // both stored halves of the kx = 0 plane: the mean of the two forms
        // (the Hermitian part, as a c2r transform takes)
        const int lm = -ky - cr.y;
        C w = cmk<C>(0.0, 0.0);
        if (lm >= 0 && lm < cr.z) {
          const C av = a[lm];
          C bv = cmk<C>(0.0, 0.0);
          if (has1) bv = b[lm];
          w.x = av.x + bv.y; w.y = bv.x - av.y;
        }
        v.x = (R)0.5 * (v.x + w.x);
        v.y = (R)0.5 * (v.y + w.y);
      }
    }
    u[n1] = v;
  }
}

// Last step of the backward y transform for the column pairs +-kx, kx in
// [x0, x0 + nkw): DFT_N1 of class m2, the two states separated, and their
// z-line rows (rstride apart) stored
// TWA: the twiddles are applied here (else the caller applied them after its
// DFT_N2 step)
template <class F, bool BAND, bool TWA, class TW>
__device__ __forceinline__ void pp_store_cols(typename F::C* row, size_t rstride, bool has1,
                                              const typename F::C* P, int ldp, const int4* col, int nkx, int x0,
                                              int nkw, int lane, const typename F::C* T, const TW& twf) {
  typedef typename F::C C;
  typedef typename F::R R;
  constexpr int N1 = F::N1, N2 = F::N2, N = F::N;
  for (int it = lane; it < nkw * N2 && lane < F::RWI; it += F::RWI) {
    const int c = it / N2, m2 = it - c * N2;
    const int mm = m2 == 0 ? 0 : N2 - m2;
    const auto tw = pp_tw(twf, T, m2);
    const int ax = x0 + c;
    C u[N1], v[N1];
    const C* pu = P + (nkx - 1 + ax) * ldp + m2;
    const C* pv = P + (nkx - 1 - ax) * ldp + mm;
    u[0] = pu[0];
#pragma unroll
    for (int k1 = 1; k1 < N1; ++k1) {
      u[k1] = pu[k1 * F::LSP];
      if (TWA) u[k1] = tw.template mul<+1>(u[k1], k1);
    }
    RDft<N1, +1>::run(u);
    // column -kx at class N2 - m2: its twiddles are exp(2 pi i k1 / N1)
    // times the conjugates of this lane's, and the first factor shifts the
    // outputs by one: element -ky of the column is output -m1 of the
    // transform with the conjugate twiddles alone (without the shift, of
    // class N2 - m2, output N1 - 1 - m1)
    v[0] = pv[0];
#pragma unroll
    for (int k1 = 1; k1 < N1; ++k1) {
      v[k1] = pv[k1 * F::LSP];
      if (TWA) v[k1] = tw.template mul<-1>(v[k1], k1);
    }
    RDft<N1, +1>::run(v);
    const int4 cr = col[ax];
    C* ra = row + cr.x;
    C* rb = ra + rstride;
#pragma unroll
    for (int m1 = 0; m1 < N1; ++m1) {
      if (F::template dead<BAND>(m1)) continue;
      const int i = m2 + N2 * m1;
      const int ky = 2 * i <= N ? i : i - N;
      const int l = ky - cr.y;
      const C e = u[m1], f0 = v[(N1 - m1) % N1], f1 = v[N1 - 1 - m1];
      const C f = TWA || m2 == 0 ? f0 : f1;
      if (l >= 0 && l < cr.z) {
        C t;
        t.x = (R)0.5 * (e.x + f.x);
        t.y = (R)0.5 * (e.y - f.y);
        ra[l] = t;
        if (has1) {
          t.x = (R)0.5 * (e.y + f.y);
          t.y = (R)-0.5 * (e.x - f.x);
          rb[l] = t;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// density pass: block (z and row split, group) runs the state pairs of its
// group through plane z
// ---------------------------------------------------------------------------
template <class F, bool BAND>
__global__ void __launch_bounds__(F::WD * 32, F::MBD)
k_pp_density(const typename F::C* __restrict__ zbuf, int nstate, int nz, int ldl, const int4* __restrict__ cols,
             int nkx, const double2* __restrict__ twg, const double* __restrict__ occ,
             double* __restrict__ rho_part, int ngroup, typename F::C* __restrict__ psir, PpSmem L,
             double* __restrict__ qpart) {
  typedef typename F::C C;
  typedef typename F::R R;
  constexpr int N1 = F::N1, N2 = F::N2, N = F::N, LDP = F::LDPD, LSP = F::LSP, LSX = F::LSX, PS = F::PS;
  constexpr int W = F::WD, RG = F::RGD, NG = F::NGD, XA = pp_ceil(RG * N2, F::RWI), XB = pp_ceil(RG * N1, 32);
  constexpr int EPC = 16 / (int)sizeof(C);  // elements per 16-byte copy
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* T = (C*)(smem_raw + L.T);
  int4* col = (int4*)(smem_raw + L.col);
  C* rows = (C*)(smem_raw + L.rows);
  C* P = (C*)(smem_raw + L.P);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int lane2 = lane % N2;  // n2 of this lane in the A steps (FIX)
  C* Sx = (C*)(smem_raw + L.S) + wid * (RG * PS);
  const int z = blockIdx.x / F::HS, h = blockIdx.x - z * F::HS, g = blockIdx.y;
  const int k1lo = h * F::K1H, k1n = min(F::K1H, N1 - k1lo);
  const int nrows = k1n * N2, r_base = k1lo * N2;
  const int npair = (nstate + 1) / 2;
  const int qb = (int)((long)g * npair / ngroup), qe = (int)((long)(g + 1) * npair / ngroup);
  const int ncol = 2 * nkx - 1;
  const int cpw = (ncol + W - 1) / W, c0 = min(wid * cpw, ncol), ncw = min(cpw, ncol - c0);
  pp_load_tw<F>(T, twg);
  for (int i = threadIdx.x; i < nkx; i += W * 32) col[i] = cols[i];
  R dens[NG][XB][N2];
#pragma unroll
  for (int a = 0; a < NG; ++a)
#pragma unroll
    for (int j = 0; j < XB; ++j)
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) dens[a][j][k2] = (R)0;
  // the z-line rows of a pair, by asynchronous copies during the x phase of
  // the pair before it
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
  for (int q = qb; q < qe; ++q) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // y phase: this warp's columns
    {
      const bool has1 = 2 * q + 1 < nstate;
      const C* rA = L.lr ? rows : zbuf + ((size_t)(2 * q) * nz + z) * ldl;
      const C* rB = L.lr ? rows + L.lr : rA + (size_t)nz * ldl;
      const PpTw<F, F::FIX> twf(T, lane2);
      for (int it = lane; it < ncw * N2 && lane < F::RWI; it += F::RWI) {
        const int c = it / N2, n2 = it - c * N2;
        const auto tw = pp_tw(twf, T, n2);
        const int kx = c0 + c - (nkx - 1);
        C u[N1];
        pp_load_col<F, BAND>(u, rA, rB, has1, col[kx < 0 ? -kx : kx], kx, n2);
        if constexpr (BAND) RDftBand<N1, -1>::run(u);
        else RDft<N1, -1>::run(u);
        C* p = P + (c0 + c) * LDP + n2;
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1)
          if (F::HS == 1 || (k1 >= k1lo && k1 < k1lo + k1n))
            p[(k1 - k1lo) * LSP] = k1 ? tw.template mul<-1>(u[k1], k1) : u[0];
      }
      __syncwarp();
      for (int it = lane; it < ncw * F::K1H; it += 32) {
        const int c = it / F::K1H, k1 = it - c * F::K1H;
        if (F::HS > 1 && k1 >= k1n) continue;
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
    // x phase: this warp's rows
    const R o0 = (R)occ[2 * q];
    const R o1 = 2 * q + 1 < nstate ? (R)occ[2 * q + 1] : (R)0;
    C* pq = psir + ((size_t)q * nz + z) * N * N + (size_t)r_base * N1;
    const PpTw<F, F::FIX> twf(T, lane2);
#pragma unroll
    for (int gi = 0; gi < NG; ++gi) {
      const int r0 = wid * F::RPD + gi * RG;
      const int nr = min(min(RG, F::RPD - gi * RG), nrows - r0);
#pragma unroll
      for (int j = 0; j < XA; ++j) {
        const int it = lane + F::RWI * j;
        const int rr = it / N2, n2 = it - rr * N2;
        if (lane < F::RWI && rr < nr) {
          const auto tw = pp_tw(twf, T, n2);
          const int r = r0 + rr, rk = r / N2;
          const C* p = P + rk * LSP + (r - rk * N2);
          C u[N1];
#pragma unroll
          for (int n1 = 0; n1 < N1; ++n1) {
            u[n1] = cmk<C>(0.0, 0.0);
            if (!F::template dead<BAND>(n1)) {
              const int k = N2 * n1 + n2;
              const int kx = 2 * k <= N ? k : k - N;
              if (kx < nkx && -kx < nkx) u[n1] = p[(kx + nkx - 1) * LDP];
            }
          }
          if constexpr (BAND) RDftBand<N1, -1>::run(u);
          else RDft<N1, -1>::run(u);
          C* sx = Sx + rr * PS + n2;
          sx[0] = u[0];
#pragma unroll
          for (int k1 = 1; k1 < N1; ++k1) sx[k1 * LSX] = tw.template mul<-1>(u[k1], k1);
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        const int it = lane + 32 * j;
        const int rr = it / N1, k1 = it - rr * N1;
        if (rr < nr) {
          C w[N2];
#pragma unroll
          for (int i = 0; i < N2; ++i) w[i] = Sx[rr * PS + k1 * LSX + i];
          RDft<N2, -1>::run(w);
          C* po = pq + (size_t)r0 * N1 + it;
#pragma unroll
          for (int k2 = 0; k2 < N2; ++k2) {
            dens[gi][j][k2] += o0 * w[k2].x * w[k2].x + o1 * w[k2].y * w[k2].y;
            __stcs(po + (size_t)k2 * (N * N1), w[k2]);
          }
        }
      }
      __syncwarp();
    }
  }
  double* out = rho_part + ((size_t)g * nz + z) * N * N;
  double qs = 0.0;  // this block's share of sum_r occ |psi(r)|^2
#pragma unroll
  for (int gi = 0; gi < NG; ++gi) {
    const int r0 = wid * F::RPD + gi * RG;
    const int nr = min(min(RG, F::RPD - gi * RG), nrows - r0);
#pragma unroll
    for (int j = 0; j < XB; ++j) {
      const int it = lane + 32 * j;
      const int rr = it / N1, k1 = it - rr * N1;
      if (rr < nr) {
        const int r = r_base + r0 + rr, rk = r / N2;
        const int y = rk + N1 * (r - rk * N2);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
          out[y * N + k1 + N1 * k2] = (double)dens[gi][j][k2];
          qs += (double)dens[gi][j][k2];
        }
      }
    }
  }
  if (qpart) {
    __shared__ double qsh[32];
    qs = block_sum(qs, qsh);
    if (threadIdx.x == 0) qpart[((size_t)g * nz + z) * F::HS + h] = qs;
  }
}

// ---------------------------------------------------------------------------
// V_KS pass from the stored psi(r): psi V_KS occ -> x^-1 -> y^-1 -> the z-line
// rows of both states
// ---------------------------------------------------------------------------
template <class F, bool BAND>
__global__ void __launch_bounds__(F::WV * 32, F::MBV)
k_pp_vks(typename F::C* __restrict__ zbuf, int nstate, int nz, int ldl, const int4* __restrict__ cols, int nkx,
         const double2* __restrict__ twg, const double* __restrict__ occ, const typename F::R* __restrict__ vks,
         int ngroup, const typename F::C* __restrict__ psir, PpSmem L) {
  typedef typename F::C C;
  typedef typename F::R R;
  constexpr int N1 = F::N1, N2 = F::N2, N = F::N, LDP = F::LDPV, LSP = F::LSP, LSX = F::LSX, PS = F::PS;
  constexpr int W = F::WV, RG = F::RGV, NG = F::NGV, XA = pp_ceil(RG * N2, F::RWI), XB = pp_ceil(RG * N1, 32);
  // FP32: V_KS of this thread's points in registers, psi(r) loaded one item ahead
  constexpr bool VREG = sizeof(R) == 4, AHEAD = sizeof(R) == 4;
  // L2 prefetch of a psi(r) pair plane in PARTS pieces (multiples of 16 bytes)
  constexpr int PARTS = (N * N * (int)sizeof(C)) % 256 == 0 ? 16 : (N * N * (int)sizeof(C)) % 64 == 0 ? 4 : 1;
  constexpr int PBYTES = N * N * (int)sizeof(C) / PARTS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* T = (C*)(smem_raw + L.T);
  int4* col = (int4*)(smem_raw + L.col);
  C* P = (C*)(smem_raw + L.P);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int lane2 = lane % N2;  // m2 of this lane in the A steps (FIX)
  C* Sx = (C*)(smem_raw + L.S) + wid * (RG * PS);
  const int z = blockIdx.x, g = blockIdx.y;
  const int npair = (nstate + 1) / 2;
  const int qb = (int)((long)g * npair / ngroup), qe = (int)((long)(g + 1) * npair / ngroup);
  const int kpw = (nkx + W - 1) / W, x0 = min(wid * kpw, nkx), nkw = min(kpw, nkx - x0);
  pp_load_tw<F>(T, twg);
  for (int i = threadIdx.x; i < nkx; i += W * 32) col[i] = cols[i];
  const R* vz = vks + (size_t)z * N * N;
  // V_KS at (row, x = k1 + N1 k2) of item it of group gi
  auto v_at = [&](int r, int k1, int k2) {
    const int rk = r / N2;
    return __ldg(vz + (rk + N1 * (r - rk * N2)) * N + k1 + N1 * k2);
  };
  R vr[VREG ? NG : 1][VREG ? XB : 1][VREG ? N2 : 1];
  if constexpr (VREG) {
#pragma unroll
    for (int gi = 0; gi < NG; ++gi) {
      const int r0 = wid * F::RPV + gi * RG;
      const int nr = min(min(RG, F::RPV - gi * RG), N - r0);
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        const int it = lane + 32 * j;
        const int rr = it / N1, k1 = it - rr * N1;
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) vr[gi][j][k2] = rr < nr ? v_at(r0 + rr, k1, k2) : (R)0;
      }
    }
  }
  // psi(r) of item s = (row group, j) of pair q -> wn
  C wn[N2];
  auto load_psi = [&](int q, int s) {
    const int gi = s / XB, j = s - gi * XB;
    const int r0 = wid * F::RPV + gi * RG;
    const int nr = min(min(RG, F::RPV - gi * RG), N - r0);
    const int it = lane + 32 * j;
    if (it < nr * N1) {
      const C* p = psir + ((size_t)q * nz + z) * N * N + (size_t)r0 * N1 + it;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) wn[k2] = __ldcs(p + (size_t)k2 * (N * N1));
    }
  };
  if (AHEAD && qb < qe) load_psi(qb, 0);
  __syncthreads();
  for (int q = qb; q < qe; ++q) {
    // the next pair's plane heads for L2 while this pair computes
    if constexpr ((N * N * (int)sizeof(C)) % (16 * PARTS) == 0) {
      if (q + 1 < qe && threadIdx.x < PARTS)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(
                         (const char*)(psir + ((size_t)(q + 1) * nz + z) * N * N) + (size_t)threadIdx.x * PBYTES),
                     "r"(PBYTES)
                     : "memory");
    }
    const bool has1 = 2 * q + 1 < nstate;
    const R o0 = (R)occ[2 * q];
    const R o1 = has1 ? (R)occ[2 * q + 1] : (R)0;
    // x phase: this warp's rows; the psi(r) of an item is loaded while the
    // item before it computes (the first one of a pair during the y phase)
    {
      const PpTw<F, F::FIX> twf(T, lane2);
#pragma unroll
      for (int gi = 0; gi < NG; ++gi) {
        const int r0 = wid * F::RPV + gi * RG;
        const int nr = min(min(RG, F::RPV - gi * RG), N - r0);
#pragma unroll
        for (int j = 0; j < XB; ++j) {
          const int it = lane + 32 * j;
          const int rr = it / N1, k1 = it - rr * N1;
          C w[N2];
          if (!AHEAD) load_psi(q, gi * XB + j);
#pragma unroll
          for (int k2 = 0; k2 < N2; ++k2) w[k2] = wn[k2];
          if (AHEAD && gi * XB + j + 1 < NG * XB) load_psi(q, gi * XB + j + 1);
          if (rr < nr) {
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) {
              R v;
              if constexpr (VREG) v = vr[gi][j][k2];
              else v = v_at(r0 + rr, k1, k2);
              w[k2].x *= v * o0;
              w[k2].y *= v * o1;
            }
            RDft<N2, +1>::run(w);
            C* sx = Sx + rr * PS + k1 * LSX;
            sx[0] = w[0];
#pragma unroll
            for (int i = 1; i < N2; ++i) sx[i] = F::FIX ? w[i] : pp_tw_inv<F>(w[i], T, i, k1);
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < XA; ++j) {
          const int it = lane + F::RWI * j;
          const int rr = it / N2, m2 = it - rr * N2;
          if (lane < F::RWI && rr < nr) {
            const auto tw = pp_tw(twf, T, m2);
            C u[N1];
            const C* sx = Sx + rr * PS + m2;
            u[0] = sx[0];
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) {
              u[k1] = sx[k1 * LSX];
              if (F::FIX) u[k1] = tw.template mul<+1>(u[k1], k1);
            }
            RDft<N1, +1>::run(u);
            const int r = r0 + rr, rk = r / N2;
            C* p = P + rk * LSP + (r - rk * N2);
#pragma unroll
            for (int m1 = 0; m1 < N1; ++m1) {
              if (F::template dead<BAND>(m1)) continue;
              const int k = m2 + N2 * m1;
              const int kx = 2 * k <= N ? k : k - N;
              if (kx < nkx && -kx < nkx) p[(kx + nkx - 1) * LDP] = u[m1];
            }
          }
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if (AHEAD && q + 1 < qe) load_psi(q + 1, 0);
    // y phase: this warp's column pairs +-kx
    for (int it = lane; it < 2 * nkw * N1; it += 32) {
      const int c = it / N1, k1 = it - c * N1;
      const int ax = x0 + (c >> 1);
      const bool neg = c & 1;
      if (neg && ax == 0) continue;
      C* p = P + (nkx - 1 + (neg ? -ax : ax)) * LDP + k1 * LSP;
      C w[N2];
#pragma unroll
      for (int i = 0; i < N2; ++i) w[i] = p[i];
      RDft<N2, +1>::run(w);
      p[0] = w[0];
#pragma unroll
      for (int i = 1; i < N2; ++i) p[i] = F::FIX ? w[i] : pp_tw_inv<F>(w[i], T, i, k1);
    }
    __syncwarp();
    {
      const PpTw<F, F::FIX> twf(T, lane2);
      pp_store_cols<F, BAND, F::FIX>(zbuf + ((size_t)(2 * q) * nz + z) * ldl, (size_t)nz * ldl, has1, P, LDP, col, nkx, x0,
                             nkw, lane, T, twf);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// shared-memory layout of one kernel; total = 0 when it does not fit
template <class F>
static PpSmem pp_layout(int mode, int nkx, int nlines) {
  typedef typename F::C C;
  constexpr int EPC = 16 / (int)sizeof(C);
  auto make = [&](bool staged) {
    PpSmem L;
    size_t o = 0;
    L.lr = staged ? (nlines + EPC - 1) / EPC * EPC : 0;
    L.T = o; o += align_up((size_t)F::N2 * F::TP * sizeof(C), 16);
    L.col = o; o += align_up((size_t)nkx * sizeof(int4), 16);
    L.rows = o; o += align_up((size_t)2 * L.lr * sizeof(C), 16);
    L.P = o; o += align_up((size_t)(2 * nkx - 1) * (mode == 0 ? F::LDPD : F::LDPV) * sizeof(C), 16);
    L.S = o; o += align_up((size_t)(mode == 0 ? F::WD * F::RGD : F::WV * F::RGV) * F::PS * sizeof(C), 16);
    L.total = o;
    return L;
  };
  PpSmem L = make(mode == 0);
  // z-line rows staged in shared memory unless that is what does not fit
  if (L.total > (size_t)OA_MAX_SMEM - 512 && mode == 0) L = make(false);
  if (L.total > (size_t)OA_MAX_SMEM - 512) L.total = 0;
  return L;
}

template <class F>
static cudaError_t pp_run(const PpArgs& A) {
  typedef typename F::C C;
  typedef typename F::R R;
  // a column and its mirror must be distinct, with no Nyquist term
  if (2 * (A.nkx - 1) >= F::N || (A.ldl & 1)) return cudaErrorNotSupported;
  const PpSmem L0 = pp_layout<F>(0, A.nkx, A.nlines), L4 = pp_layout<F>(4, A.nkx, A.nlines);
  if (!L0.total || !L4.total) return cudaErrorNotSupported;
  const bool band = F::CANBAND && 4 * (A.nkx - 1) < F::N && 4 * A.kymax < F::N;
  auto density = [&](auto kern) -> cudaError_t {
    const cudaError_t e = oa_smem_limit(kern);
    if (e != cudaSuccess) return e;
    if (A.mode < 0) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(A.dbps, kern, F::WD * 32, L0.total);
    kern<<<dim3(A.nz * F::HS, A.ngroup), F::WD * 32, L0.total, A.st>>>(
        (const C*)A.zbuf, A.nstate, A.nz, A.ldl, (const int4*)A.cols, A.nkx, A.tw, A.occ, A.rho_part, A.ngroup,
        (C*)A.psir, L0, A.qpart);
    return cudaGetLastError();
  };
  auto vks = [&](auto kern) -> cudaError_t {
    const cudaError_t e = oa_smem_limit(kern);
    if (e != cudaSuccess) return e;
    if (A.mode < 0) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(A.vbps, kern, F::WV * 32, L4.total);
    kern<<<dim3(A.nz, A.ngroup), F::WV * 32, L4.total, A.st>>>((C*)A.zbuf, A.nstate, A.nz, A.ldl,
                                                               (const int4*)A.cols, A.nkx, A.tw, A.occ,
                                                               (const R*)A.vks, A.ngroup, (const C*)A.psir, L4);
    return cudaGetLastError();
  };
  auto run = [&](auto kd, auto kv) -> cudaError_t {
    if (A.mode < 0) {
      *A.split = F::HS;
      const cudaError_t e = density(kd);
      return e != cudaSuccess ? e : vks(kv);
    }
    return A.mode == 0 ? density(kd) : vks(kv);
  };
  if constexpr (F::CANBAND) {
    if (band) return run(k_pp_density<F, true>, k_pp_vks<F, true>);
  }
  return run(k_pp_density<F, false>, k_pp_vks<F, false>);
}
