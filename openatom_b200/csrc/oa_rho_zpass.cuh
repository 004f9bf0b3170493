// z pass of the density path (oa_rho.cu launches it): FFT(-) -> Hartree + local
// pseudopotential + Ewald (recip) in G -> FFT(+), LB z-lines per block.
//
// The structure factors S_t(g) = sum_{a in t} e^{i g.R_a} factorise per
// z-line: w[line][a] = e^{i (gx x_a + gy y_a)} is formed once per block in
// shared memory (atoms grouped by type, each group padded to a multiple of
// four with zeros), and S is the product of w [line][atom] and the z phases
// [atom][kz].  Of the complex product the four real ones Re w Re z, Im w Im z,
// Re w Im z, Im w Re z run on the FP64 tensor cores (8 lines x 8 kz tiles),
// and their sums and differences give S at kz and at -kz.  A thread per point
// was bound by the latency of its z-phase loads (two points per load).
// Measured before -> now: 108^3 with 96 atoms 82 -> 58 us, 120^3 with 192 atoms
// 196 (runtime transforms) -> 78 us, 160^3 with 384 atoms 1050 -> 611 us beside the
// nonlocal branch, 64^3 with 24 atoms 17 -> 11 us.
#pragma once
#include "oa_rho_common.cuh"
#include "oa_rdft.cuh"
#include "oa_lengths.h"

struct RhoTypeOff { int off[5]; };

// Lines per block: the eight rows of a tile (twice the blocks of sixteen, for
// the small grids and an even last wave).  With forces sixteen, since the ion
// step sums the blocks' partials one after the other.
template <bool FORCES> struct RhoZLB { static constexpr int value = FORCES ? 16 : 8; };

__device__ __forceinline__ void rho_dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

// FORCES: also the atom forces of the local pseudopotential and the
// reciprocal Ewald sum (CP_hart_eext_calc's force loop, cp_hart_ext.C:300-360):
// per g of the block the per-type coefficients
//   A_t = w (Re rho v_t + Re S_q ewf q_t),  B_t = w (-Im rho v_t + Im S_q ewf q_t)
// go to shared memory, then one warp per atom sums
//   F_a += g (A_t Im h_a - B_t Re h_a),  h_a = e^{i g.R_a},
// over the block's g-points into fpart[block][atom][3].
// EES (ees.zq set; eesHartEextGchare / eesEwaldGchare, cp_hart_ext.C:1005-1340):
// the per-type structure factors are b(g) Qhat_t(g), Qhat_t taken from the
// transformed B-spline grids (types 2k, 2k+1 split from complex grid k by
// the conjugate point -g); FORCES writes the per-type force transforms
//   Y_t = v_t conj(rho b) + q_t ewf conj(b) S_q
// (the Ewald part folded in by the type's charge) into ees.zy at g and, for
// kx > 0, their conjugates at -g, instead of reducing over atoms here.
template <int N1, int N2, bool FORCES>
__global__ void __launch_bounds__(OA_NTHREADS, 2)
k_rho_zpass(double2* __restrict__ dz, int ldl_d, int nlines_d, int nx, int ny, int nz,
            OaFftPlan pz, const double2* __restrict__ twz,
            double tpi_l, double vol, double ecut4, double falp2, double gz_term,
            int natm, int ntype, const int* __restrict__ atm_perm, RhoTypeOff toff, RhoTypeOff poff, int ldp,
            const double* __restrict__ q_type, const double2* __restrict__ phase, int ktab,
            const double* __restrict__ spl, int nspl, double gmin, double dg,
            double* __restrict__ part, double* __restrict__ fpart, EesLocArgs ees) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LB = RhoZLB<FORCES>::value;
  const int ldz = nz + 1;
  const bool use_ees = ees.zq != nullptr;
  constexpr bool TP = N1 > 0;  // two-pass compile-time transforms
  const int ldb = TP ? (ZLd<N1, N2>::PS > ldz ? ZLd<N1, N2>::PS : ldz) : ldz;
  double2* tw = (double2*)smem_raw;
  double2* a = tw + align_up_r(nz, 2);
  double2* b = a + LB * ldz;
  double2* pxy = b + LB * ldb;         // [LB][ldp], padded type order
  int* zoff = (int*)(pxy + LB * ldp);  // [ldp]: z-phase row of a padded atom
  __shared__ double sh[3 * 32];
  const int l0 = blockIdx.x * LB;
  const int nb = min(LB, nlines_d - l0);
  const int nt = 2 * ktab + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  // blocks without a line inside the density sphere only write zeros
  bool in = false;
  if (lane < nb) {
    const int kx = (l0 + lane) / ny;
    int ky = l0 + lane - kx * ny; if (2 * ky >= ny) ky -= ny;
    const double gx = tpi_l * kx, gy = tpi_l * ky;
    in = kx <= ktab && abs(ky) <= ktab && gx * gx + gy * gy <= ecut4;
  }
  if (!__any_sync(0xffffffffu, in)) {
    for (int idx = threadIdx.x; idx < nz * LB; idx += blockDim.x) {
      const int zz = idx / LB, lb = idx - zz * LB;
      if (lb < nb) dz[(size_t)zz * ldl_d + l0 + lb] = make_double2(0.0, 0.0);
    }
    if (FORCES && !use_ees)
      for (int i = threadIdx.x; i < 3 * natm; i += blockDim.x) fpart[(size_t)blockIdx.x * 3 * natm + i] = 0.0;
    if (threadIdx.x < 3) part[3 * blockIdx.x + threadIdx.x] = 0.0;
    return;
  }
  load_twiddles(tw, twz, nz);
  // FORCES: per-type (A, B) coefficients, the first type's in the buffer that
  // the transforms leave free (row stride ldz), the others' after zoff
  double2* cf = (double2*)(smem_raw + (((size_t)((char*)(zoff + ldp) - (char*)smem_raw) + 15) & ~(size_t)15));
  // the density coefficients of the block's lines: every 16-byte copy
  // issued before any is waited for
  for (int idx = threadIdx.x; idx < nz * LB; idx += blockDim.x) {
    const int zz = idx / LB, lb = idx - zz * LB;
    if (lb < nb) rho_cp16(a + lb * ldz + zz, dz + (size_t)zz * ldl_d + l0 + lb);
  }
  rho_cp_commit();
  if (!use_ees) {
    const int np = poff.off[ntype];
    for (int idx = threadIdx.x; idx < LB * np; idx += blockDim.x) {
      const int lb = idx / np, p = idx - lb * np;
      int t = 0;
      while (t + 1 < ntype && p >= poff.off[t + 1]) ++t;
      const int ia = toff.off[t] + p - poff.off[t];
      const bool pad = ia >= toff.off[t + 1];
      const int at = pad ? 0 : atm_perm[ia];
      const int l = l0 + lb;
      const int kx = l / ny;
      int ky = l - kx * ny; if (2 * ky >= ny) ky -= ny;
      double2 v = make_double2(0.0, 0.0);
      if (!pad && lb < nb && kx <= ktab && abs(ky) <= ktab) {
        const double2* ph = phase + (size_t)at * 3 * nt;
        v = cmul(ph[kx + ktab], ph[nt + ky + ktab]);
      }
      pxy[lb * ldp + p] = v;
      if (lb == 0) zoff[p] = (at * 3 + 2) * nt + ktab;
    }
  }
  rho_cp_wait();
  __syncthreads();
  double2* r;
  if constexpr (TP) {
    zfft2<N1, N2, -1>(a, b, ldz, nb, tw);
    r = a;
  } else {
    r = fft_pingpong<-1>(a, b, ldz, nb, pz, tw);
  }
  double2* cf0 = r == a ? b : a;
  const double pi = 3.14159265358979323846;
  const double fpi = 4.0 * pi;
  double acc[3] = {0.0, 0.0, 0.0};
  // One warp per tile of 8 lines x 8 kz: lane (li, q) holds line li and
  // kz = k0 + 2 q + {0, 1}, each at +kz and -kz
  const int li = lane >> 2, q = lane & 3;
  for (int tile = warp;; tile += nwarp) {
    const int kt = tile / (LB / 8), mt = tile - kt * (LB / 8), k0 = kt * 8;
    if (2 * k0 > nz) break;
    const int lb = mt * 8 + li, l = l0 + lb;
    const int kx = l / ny;
    int ky = l - kx * ny; if (2 * ky >= ny) ky -= ny;
    const bool kok = lb < nb && kx <= ktab && abs(ky) <= ktab;
    const double gx = tpi_l * kx, gy = tpi_l * ky;
    double g2[2], hh[2];
    int cls[2], ii[2];  // cls: 0 outside, 1 g = 0, 2 inside the density sphere
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int kz = k0 + 2 * q + e;
      const double gz = tpi_l * kz;
      g2[e] = gx * gx + gy * gy + gz * gz;
      cls[e] = 0; ii[e] = 1; hh[e] = 0.0;
      if (lb < nb && g2[e] == 0.0) cls[e] = 1;
      else if (kok && kz <= ktab && 2 * kz <= nz && g2[e] <= ecut4) {
        cls[e] = 2;
        // spline interval of the local pseudopotential (CP_get_vpsnow, cp_hart_ext.C:433-480)
        const double g = sqrt(g2[e]);
        int i1 = (int)((g - gmin) / dg + 1.0);
        i1 = min(i1, nspl); i1 = max(i1, 1);
        ii[e] = i1;
        hh[e] = g - ((double)(i1 - 1) * dg + gmin);
      }
    }
    // v_t(|g|) / V
    auto vloc = [&](int t, int e) {
      const double* cc = spl + ((size_t)t * nspl + (ii[e] - 1)) * 4;
      return (((cc[3] * hh[e] + cc[2]) * hh[e] + cc[1]) * hh[e] + cc[0]) / vol;
    };
    // sign s: 0 kz, 1 -kz (its own point unless kz = 0; at 2 kz = nz the only one)
    auto zpt = [&](int e, int s) {
      const int kz = k0 + 2 * q + e;
      return s == 0 ? (2 * kz < nz ? kz : -1) : (kz > 0 && 2 * kz <= nz ? nz - kz : -1);
    };
    // EES grid offsets of g (m = 0) and -g (m = 1); |k| <= ktab < n / 2 there
    auto eoff = [&](int e, int s, int m) {
      const int kz = s ? -(k0 + 2 * q + e) : k0 + 2 * q + e;
      const int jx = m ? -kx : kx, jy = m ? -ky : ky, jz = m ? -kz : kz;
      return ((size_t)(jz < 0 ? jz + ees.nc : jz) * ees.nb + (jy < 0 ? jy + ees.nb : jy)) * ees.na +
             (jx < 0 ? jx + ees.na : jx);
    };
    auto ebg = [&](int e, int s) {
      const int kz = s ? -(k0 + 2 * q + e) : k0 + 2 * q + e;
      return cmul(cmul(ees.ba[kx], ees.bb[ky < 0 ? ky + ees.nb : ky]), ees.bc[kz < 0 ? kz + ees.nc : kz]);
    };
    double2 sfq[2][2], vext[2][2];  // [e][s]: Ewald charge sum sum_t q_t S_t, V_ext = sum_t S_t v_t / V
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int s = 0; s < 2; ++s) sfq[e][s] = vext[e][s] = make_double2(0.0, 0.0);
    if (__any_sync(0xffffffffu, cls[0] == 2 || cls[1] == 2)) {
      for (int t = 0; t < ntype && t < 4; ++t) {
        double2 st[2][2];
        if (use_ees) {
          // Qhat_t = (Z +- conj Z(-g)) / (2 or 2i) of grid t / 2, times b(g)
          const double2* zg = ees.zq + (size_t)(t >> 1) * ees.gstride;
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              st[e][s] = make_double2(0.0, 0.0);
              if (cls[e] != 2) continue;
              const double2 z = zg[eoff(e, s, 0)], zm = zg[eoff(e, s, 1)];
              const double2 qh = (t & 1) ? make_double2(0.5 * (z.y + zm.y), 0.5 * (zm.x - z.x))
                                         : make_double2(0.5 * (z.x + zm.x), 0.5 * (z.y - zm.y));
              st[e][s] = cmul(ebg(e, s), qh);
            }
        } else {
          double rr[2] = {0.0, 0.0}, im[2] = {0.0, 0.0}, ri[2] = {0.0, 0.0}, ir[2] = {0.0, 0.0};
          const double2* w = pxy + lb * ldp + q;
          const double2* zp = phase + min(k0 + li, ktab);
#pragma unroll 4
          for (int p = poff.off[t]; p < poff.off[t + 1]; p += 4) {
            const double2 wv = w[p], zv = zp[zoff[p + q]];
            rho_dmma(rr, wv.x, zv.x);
            rho_dmma(im, wv.y, zv.y);
            rho_dmma(ri, wv.x, zv.y);
            rho_dmma(ir, wv.y, zv.x);
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            st[e][0] = make_double2(rr[e] - im[e], ri[e] + ir[e]);
            st[e][1] = make_double2(rr[e] + im[e], ir[e] - ri[e]);
          }
        }
        const double qa = q_type[t];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (cls[e] != 2) continue;
          const double vt = vloc(t, e);
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            sfq[e][s].x += qa * st[e][s].x; sfq[e][s].y += qa * st[e][s].y;
            vext[e][s].x += st[e][s].x * vt; vext[e][s].y += st[e][s].y * vt;
          }
        }
      }
    }
    const double wn = kx == 0 ? 1.0 : 2.0;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      double hf = 0.0, ewf = 0.0;
      if (cls[e] == 2) {
        hf = fpi / (g2[e] * vol);
        ewf = fpi * exp(-g2[e] / falp2) / (g2[e] * vol);
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int zz = zpt(e, s);
        if (lb >= nb || zz < 0) continue;
        const double2 rho = r[lb * ldz + zz];
        double2 out = make_double2(0.0, 0.0);
        if (cls[e] == 1) {
          double gzt = gz_term;
          if (use_ees) {
            // sum_t gzvps_t b(0) Qhat_t(0) / V (eesHartEextGchare's g = 0 branch)
            const double b0 = cmul(cmul(ees.ba[0], ees.bb[0]), ees.bc[0]).x;
            gzt = 0.0;
            for (int t = 0; t < ntype && t < 4; ++t) {
              const double2 z0 = ees.zq[(size_t)(t >> 1) * ees.gstride];
              const double yt = ees.gzvps[t] / vol * b0;
              gzt += yt * ((t & 1) ? z0.y : z0.x);
              if constexpr (FORCES) {
                double* w0 = (double*)(ees.zy + (size_t)(t >> 1) * ees.gstride);
                w0[t & 1] = yt * rho.x;
              }
            }
          }
          out.x = gzt;
          acc[1] += gzt * rho.x;
        } else if (cls[e] == 2) {
          acc[0] += hf * (rho.x * rho.x + rho.y * rho.y) * wn;
          out.x = rho.x * hf; out.y = rho.y * hf;
          acc[2] += ewf * (sfq[e][s].x * sfq[e][s].x + sfq[e][s].y * sfq[e][s].y) * wn;
          out.x += vext[e][s].x; out.y -= vext[e][s].y;            // vks += conj(vext)
          acc[1] += (rho.x * vext[e][s].x - rho.y * vext[e][s].y) * wn;  // Re(rho vext)
        }
        r[lb * ldz + zz] = out;
        if (FORCES && use_ees) {
          if (cls[e] == 2) {
            const double2 bg = ebg(e, s);
            const double2 rb = cconj(cmul(rho, bg));
            const double2 sqe = cmul(cconj(bg), sfq[e][s]);
            const bool mirror = kx > 0;
            for (int t0 = 0; t0 < ntype && t0 < 4; t0 += 2) {
              double2 y[2];
              for (int u = 0; u < 2; ++u) {
                const int t = t0 + u;
                y[u] = make_double2(0.0, 0.0);
                if (t < ntype) {
                  const double qt = q_type[t] * ewf, vt = vloc(t, e);
                  y[u].x = vt * rb.x + qt * sqe.x;
                  y[u].y = vt * rb.y + qt * sqe.y;
                }
              }
              double2* w = ees.zy + (size_t)(t0 >> 1) * ees.gstride;
              w[eoff(e, s, 0)] = make_double2(y[0].x - y[1].y, y[0].y + y[1].x);
              if (mirror) w[eoff(e, s, 1)] = make_double2(y[0].x + y[1].y, y[1].x - y[0].y);
            }
          }
        } else if constexpr (FORCES) {
          for (int t = 0; t < ntype && t < 4; ++t) {
            double2 ab = make_double2(0.0, 0.0);
            if (cls[e] == 2) {
              const double qt = q_type[t], vt = vloc(t, e);
              ab.x = wn * (rho.x * vt + sfq[e][s].x * ewf * qt);
              ab.y = wn * (-rho.y * vt + sfq[e][s].y * ewf * qt);
            }
            (t == 0 ? cf0[lb * ldz + zz] : cf[((t - 1) * LB + lb) * nz + zz]) = ab;
          }
        }
      }
    }
  }
  __syncthreads();
  if (FORCES && !use_ees) {
    // one warp per atom (type order), lanes over the block's (line, plane) points
    for (int ia = warp; ia < natm; ia += nwarp) {
      int t = 0;
      while (t + 1 < ntype && ia >= toff.off[t + 1]) ++t;
      const int p = poff.off[t] + ia - toff.off[t];
      double fx = 0.0, fy = 0.0, fz = 0.0;
      for (int e = lane; e < nb * nz; e += 32) {
        const int lb = e / nz, zz = e - lb * nz;
        const double2 ab = t == 0 ? cf0[lb * ldz + zz] : cf[((t - 1) * LB + lb) * nz + zz];
        if (ab.x == 0.0 && ab.y == 0.0) continue;
        const int l = l0 + lb;
        const int kx = l / ny;
        int ky = l - kx * ny; if (2 * ky >= ny) ky -= ny;
        int kz = zz; if (2 * kz >= nz) kz -= nz;
        const double2 h = cmul(pxy[lb * ldp + p], phase[zoff[p] + kz]);
        const double comp = ab.x * h.y - ab.y * h.x;
        fx += tpi_l * kx * comp;
        fy += tpi_l * ky * comp;
        fz += tpi_l * kz * comp;
      }
      fx = warp_sum_d(fx);
      fy = warp_sum_d(fy);
      fz = warp_sum_d(fz);
      if (lane == 0) {
        double* o = fpart + ((size_t)blockIdx.x * natm + atm_perm[ia]) * 3;
        o[0] = fx; o[1] = fy; o[2] = fz;
      }
    }
    __syncthreads();  // cf0 is the buffer that the inverse transform writes first
  }
  double2* r2;
  if constexpr (TP) {
    zfft2<N1, N2, +1>(a, b, ldz, nb, tw);
    r2 = a;
  } else {
    double2* other = (r == a) ? b : a;
    r2 = fft_pingpong<+1>(r, other, ldz, nb, pz, tw);
  }
  for (int idx = threadIdx.x; idx < nz * LB; idx += blockDim.x) {
    const int zz = idx / LB, lb = idx - zz * LB;
    if (lb < nb) dz[(size_t)zz * ldl_d + l0 + lb] = r2[lb * ldz + zz];
  }
  block_sum_n<3>(acc, sh);
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x + 0] = acc[0];
    part[3 * blockIdx.x + 1] = acc[1];
    part[3 * blockIdx.x + 2] = acc[2];
  }
}

template <bool FORCES> cudaError_t rho_zpass(oa_ctx* c, cudaStream_t s, int nblk, double* part, double* fpart,
                                             const EesLocArgs& ees) {
  constexpr int LB = RhoZLB<FORCES>::value;
  const double tpi_l = 2.0 * 3.14159265358979323846 / c->box;
  RhoTypeOff toff, poff;
  for (int t = 0; t < 5; ++t) toff.off[t] = c->type_off[t];
  poff.off[0] = 0;
  for (int t = 0; t < 4; ++t) poff.off[t + 1] = poff.off[t] + (t < c->ntype ? (toff.off[t + 1] - toff.off[t] + 3) / 4 * 4 : 0);
  // row stride 4 mod 8: a tile's loads of w fall on different banks
  int ldp = poff.off[4];
  if (ldp % 8 == 0) ldp += 4;
  auto go = [&](auto kern, int ldb) -> cudaError_t {
    size_t sm = (align_up_r(c->nz, 2) + (size_t)LB * (c->nz + 1) + (size_t)LB * ldb + (size_t)LB * ldp) *
                    sizeof(double2) + (size_t)ldp * sizeof(int);  // zoff
    if (FORCES) sm = align_up_r(sm, 16) + (size_t)LB * c->nz * (c->ntype - 1) * sizeof(double2);
    if (sm > (size_t)OA_MAX_SMEM) return cudaErrorNotSupported;
    cudaError_t e = oa_smem_limit(kern);
    if (e != cudaSuccess) return e;
    kern<<<nblk, OA_NTHREADS, sm, s>>>((double2*)c->dz, c->ldl_d, c->nlines_d, c->nx, c->ny, c->nz, c->plan_z,
                                       c->tw_z, tpi_l, c->vol, c->ecut_rho, 4.0 * c->alp_ewd * c->alp_ewd,
                                       c->gzvps_sum / c->vol, c->natm, c->ntype, c->atm_perm, toff, poff, ldp,
                                       c->q_type, c->phase, c->kmax_tab, c->spl, c->nspl, c->spl_gmin, c->spl_dg,
                                       part, fpart, ees);
    return cudaGetLastError();
  };
  cudaError_t e = cudaErrorNotSupported;
  switch (c->nz) {
#define OA_ZP(NN, A, B) \
  case NN: e = go(k_rho_zpass<A, B, FORCES>, ZLd<A, B>::PS > c->nz + 1 ? ZLd<A, B>::PS : c->nz + 1); break;
    OA_LENGTHS_ALL(OA_ZP)
#undef OA_ZP
    default: break;
  }
  if (e == cudaErrorNotSupported) e = go(k_rho_zpass<0, 0, FORCES>, c->nz + 1);
  return e;
}
