// Density -> V_KS(r) on one GPU (FP64 in both precision forms; it is one
// grid per step against 2 N_state state transforms).
//
// Replaces:
//   CP_Rho_RealSpacePlane::acceptDensity/handleDensityReduction (CP_Rho_RealSpacePlane.C:398-520)
//     sum of state-group partial densities, probScale = 1/V         -> k_rho_xc
//   CPXCFNCTS::CP_exc_calc (cp_pz_lda.C:23-175), energyComputation (:739) -> k_rho_xc
//   fftRhoRtoRhoG (:831) + Charm forward FFT, rho * volumeFactor   -> k_rho_plane_fwd + k_rho_zpass
//   CP_Rho_GHartExt::HartExtVksG (CP_Rho_GHartExt.C:461) ->
//     CPLOCAL::CP_hart_eext_calc (cp_hart_ext.C:56-431)             -> k_rho_zpass
//   FFTVks (CP_Rho_GHartExt.C:532) + acceptHartVks (CP_Rho_RealSpacePlane.C:1365) -> k_rho_zpass + k_rho_plane_bwd
// Charm-FFT's sign convention is not in the tree; forward exp(-i g.r) and
// backward exp(+i g.r) are the ones under which the e^{+i g.R} structure
// factor of cp_hart_ext.C gives E_ext = integral rho V_loc.
#include "oa_internal.h"
#include "oa_rdft.cuh"
#include "oa_rho_common.cuh"
#include "oa_lengths.h"

// ---------------------------------------------------------------------------
// density sum + PZ-LDA
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(OA_NTHREADS)
k_rho_xc(const double* __restrict__ rho_part, int ngroup, size_t npts, double rvol, double cfac,
         const double* __restrict__ qscale, double* __restrict__ rho, double* __restrict__ vxc,
         double* __restrict__ part) {
  // cfac = 0 drops the PZ correlation (LYP correlation on, cp_pz_lda.C:66);
  // qscale (mixed form): the renormalisation to the exact electron count
  if (qscale) rvol *= qscale[0];
  __shared__ double sh[3 * 32];
  // Perdew-Zunger constants (cp_pz_lda.C:46-52)
  const double gamma = -0.14230, beta1 = 1.05290, beta2 = 0.33340;
  const double au = 0.03110, bu = -0.0480, cu = 0.00200, du = -0.01160;
  const double power = 1.0 / 3.0;
  const double rat1 = (7.0 / 6.0) * beta1, rat2 = (4.0 / 3.0) * beta2;
  const double pi = 3.14159265358979323846, fpi = 4.0 * pi;
  // rs = (3 / (4 pi r))^(1/3) and -(3 r / pi)^(1/3) from one cube root of
  // r; a negative density gives NaN as the powers do
  const double c_rs = cbrt(3.0 / fpi), c_x = cbrt(3.0 / pi);
  double acc[3] = {0.0, 0.0, 0.0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < npts; i += (size_t)gridDim.x * blockDim.x) {
    double r = 0.0;
    for (int g = 0; g < ngroup; ++g) r += rho_part[(size_t)g * npts + i];
    r *= rvol;
    rho[i] = r;
    const double cr = r >= 0.0 ? cbrt(r) : __longlong_as_double(0x7ff8000000000000LL);
    const double rs = c_rs / cr;
    const double sqtrs = sqrt(rs);
    const double xfact = -c_x * cr;
    double cfact, mufact;
    if (rs >= 1.0) {
      const double cf1 = 1.0 + beta1 * sqtrs + beta2 * rs;
      const double cf2 = 1.0 + rat1 * sqtrs + rat2 * rs;
      cfact = gamma / cf1;
      mufact = cfact * (cf2 / cf1);
    } else {
      const double lnrs = log(rs);
      cfact = au * lnrs + bu + cu * rs * lnrs + du * rs;
      mufact = au * lnrs + (bu - power * au) + 2.0 * power * cu * rs * lnrs + power * (2.0 * du - cu) * rs;
    }
    cfact *= cfac;
    mufact *= cfac;
    acc[0] += xfact * r;
    acc[1] += cfact * r;
    const double v = xfact + mufact;
    acc[2] += v * r;
    vxc[i] = v;
  }
  block_sum_n<3>(acc, sh);
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x + 0] = acc[0];
    part[3 * blockIdx.x + 1] = acc[1];
    part[3 * blockIdx.x + 2] = acc[2];
  }
}

// ---------------------------------------------------------------------------
// plane helpers for the dense density grid (nkx = nx/2 + 1 columns)
// ---------------------------------------------------------------------------
template <typename C>
__device__ __forceinline__ C herm_xd(const C* P, int ldy, int nkx, int nx, int k, int y) {
  C v = cmk<C>(0.0, 0.0);
  if (k <= nx / 2) {
    if (k < nkx) v = P[k * ldy + y];
    if (k == 0 || 2 * k == nx) v.y = 0;
  } else {
    const int kk = nx - k;
    if (kk < nkx) v = cconj(P[kk * ldy + y]);
  }
  return v;
}

struct RhoPlaneSmem { size_t tw_x, tw_y, P, W1, W2, total; };

static RhoPlaneSmem rho_plane_layout(int nx, int ny, int nkx, int npair, int ychunk) {
  RhoPlaneSmem L;
  const int ldx = nx + 1, ldy = ny + 1;
  size_t o = 0;
  L.tw_x = o; o += align_up_r(nx * sizeof(double2), 16);
  L.tw_y = o; o += align_up_r(ny * sizeof(double2), 16);
  L.P = o; o += align_up_r((size_t)nkx * ldy * sizeof(double2), 16);
  size_t wsz = (size_t)npair * ldx;
  if ((size_t)ychunk * ldy > wsz) wsz = (size_t)ychunk * ldy;
  L.W1 = o; o += align_up_r(wsz * sizeof(double2), 16);
  L.W2 = o; o += align_up_r(wsz * sizeof(double2), 16);
  L.total = o;
  return L;
}

// forward: rho(x,y,z) * V/N -> r2c x (-) by row pairs -> y FFT (-) -> dz[z][k*ny+y]
__global__ void __launch_bounds__(OA_NTHREADS)
k_rho_plane_fwd(const double* __restrict__ rho, double scale, int nx, int ny, int nz, int nkx,
                OaFftPlan px, OaFftPlan py, const double2* __restrict__ twx, const double2* __restrict__ twy,
                double2* __restrict__ dz, int ldl_d, int npair, int ychunk, RhoPlaneSmem L, size_t fin,
                size_t fout) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* stwx = (double2*)(smem_raw + L.tw_x);
  double2* stwy = (double2*)(smem_raw + L.tw_y);
  double2* P = (double2*)(smem_raw + L.P);
  double2* W1 = (double2*)(smem_raw + L.W1);
  double2* W2 = (double2*)(smem_raw + L.W2);
  const int ldx = nx + 1, ldy = ny + 1;
  const int z = blockIdx.x;
  const int npairs = (ny + 1) / 2;
  rho += blockIdx.y * fin;
  dz += blockIdx.y * fout;
  load_twiddles(stwx, twx, nx);
  load_twiddles(stwy, twy, ny);
  const double* rz = rho + (size_t)z * nx * ny;
  for (int p0 = 0; p0 < npairs; p0 += npair) {
    const int np = min(npair, npairs - p0);
    __syncthreads();
    for (int idx = threadIdx.x; idx < np * nx; idx += blockDim.x) {
      const int p = idx / nx, x = idx - p * nx;
      const int y1 = 2 * (p0 + p), y2 = y1 + 1;
      W1[p * ldx + x] = make_double2(rz[y1 * nx + x] * scale, (y2 < ny) ? rz[y2 * nx + x] * scale : 0.0);
    }
    __syncthreads();
    double2* r = fft_pingpong<-1>(W1, W2, ldx, np, px, stwx);
    for (int idx = threadIdx.x; idx < np * nkx; idx += blockDim.x) {
      const int p = idx / nkx, k = idx - p * nkx;
      const int y1 = 2 * (p0 + p), y2 = y1 + 1;
      const double2 a = r[p * ldx + k];
      const double2 b = cconj(r[p * ldx + (k == 0 ? 0 : nx - k)]);
      P[k * ldy + y1] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
      if (y2 < ny) P[k * ldy + y2] = make_double2(0.5 * (a.y - b.y), -0.5 * (a.x - b.x));
    }
  }
  __syncthreads();
  for (int c0 = 0; c0 < nkx; c0 += ychunk) {
    const int nb = min(ychunk, nkx - c0);
    fft_inout<-1>(P + c0 * ldy, ldy, P + c0 * ldy, ldy, W1, W2, ldy, nb, py, stwy);
  }
  double2* out = dz + (size_t)z * ldl_d;
  for (int idx = threadIdx.x; idx < nkx * ny; idx += blockDim.x) {
    const int k = idx / ny, y = idx - k * ny;
    out[idx] = P[k * ldy + y];
  }
}

// backward: dz[z][k*ny+y] -> y FFT (+) -> c2r x (+) -> vks = V + vxc
template <typename R>
__global__ void __launch_bounds__(OA_NTHREADS)
k_rho_plane_bwd(const double2* __restrict__ dz, int ldl_d, int nx, int ny, int nz, int nkx,
                OaFftPlan px, OaFftPlan py, const double2* __restrict__ twx, const double2* __restrict__ twy,
                const double* __restrict__ vxc, R* __restrict__ vks, int npair, int ychunk, RhoPlaneSmem L,
                size_t fin, size_t fout) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* stwx = (double2*)(smem_raw + L.tw_x);
  double2* stwy = (double2*)(smem_raw + L.tw_y);
  double2* P = (double2*)(smem_raw + L.P);
  double2* W1 = (double2*)(smem_raw + L.W1);
  double2* W2 = (double2*)(smem_raw + L.W2);
  const int ldx = nx + 1, ldy = ny + 1;
  const int z = blockIdx.x;
  const int npairs = (ny + 1) / 2;
  dz += blockIdx.y * fin;
  vks += blockIdx.y * fout;
  load_twiddles(stwx, twx, nx);
  load_twiddles(stwy, twy, ny);
  const double2* in = dz + (size_t)z * ldl_d;
  for (int idx = threadIdx.x; idx < nkx * ny; idx += blockDim.x) {
    const int k = idx / ny, y = idx - k * ny;
    P[k * ldy + y] = in[idx];
  }
  __syncthreads();
  for (int c0 = 0; c0 < nkx; c0 += ychunk) {
    const int nb = min(ychunk, nkx - c0);
    fft_inout<+1>(P + c0 * ldy, ldy, P + c0 * ldy, ldy, W1, W2, ldy, nb, py, stwy);
  }
  const double* vz = vxc ? vxc + (size_t)z * nx * ny : nullptr;  // null: vks = V
  R* oz = vks + (size_t)z * nx * ny;
  for (int p0 = 0; p0 < npairs; p0 += npair) {
    const int np = min(npair, npairs - p0);
    for (int idx = threadIdx.x; idx < np * nx; idx += blockDim.x) {
      const int p = idx / nx, k = idx - p * nx;
      const int y1 = 2 * (p0 + p), y2 = y1 + 1;
      const double2 a = herm_xd(P, ldy, nkx, nx, k, y1);
      double2 b = make_double2(0.0, 0.0);
      if (y2 < ny) b = herm_xd(P, ldy, nkx, nx, k, y2);
      W1[p * ldx + k] = make_double2(a.x - b.y, a.y + b.x);
    }
    __syncthreads();
    double2* r = fft_pingpong<+1>(W1, W2, ldx, np, px, stwx);
    for (int idx = threadIdx.x; idx < np * nx; idx += blockDim.x) {
      const int p = idx / nx, x = idx - p * nx;
      const int y1 = 2 * (p0 + p), y2 = y1 + 1;
      const double2 v = r[p * ldx + x];
      oz[y1 * nx + x] = (R)(v.x + (vz ? vz[y1 * nx + x] : 0.0));
      if (y2 < ny) oz[y2 * nx + x] = (R)(v.y + (vz ? vz[y2 * nx + x] : 0.0));
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// BLYP gradient correction (cp_grad_rho_ctrl.C, cp_becke.C; the driver's
// divRhoVksGspace / acceptGradRhoVks / whiteByrdFFT / acceptWhiteByrd,
// CP_Rho_GSpacePlane.C:278-380, CP_Rho_RealSpacePlane.C:1061-1350):
//   k_rho_grad_z   rho(g) -> i g_a rho(g) / V on the density sphere, z^-1
//   (x-y inverse)  -> grad rho(r), three fields
//   k_rho_gga      per point: EGGA density, vxc += df/drho,
//                  h = df/d|grad rho| grad rho / |grad rho|
//   (x-y forward of h / N)
//   k_rho_div_z    z forward of h, i g . h(g) on the sphere, z^-1, and
//                  subtracted from the V_KS z-lines before their x-y inverse
// ---------------------------------------------------------------------------
struct GgaTerm { double f, dfr, dfg; };

// Becke 88 correction to the LDA exchange, spin-unpolarised (becke_gcx_lda,
// cp_becke.C:21-88): per spin rho_s = rho / 2, x = (g / 2) / rho_s^(4/3),
// b = x^2 / (1 + 6 beta x asinh x), f = -2 beta rho_s^(4/3) b;
// df/drho = -(4/3) beta rho_s^(1/3) (b - x b'), df/dg = -beta b'.
__device__ __forceinline__ GgaTerm gga_becke88(double rho, double g) {
  const double beta = 0.0042;
  const double rs = 0.5 * rho;
  const double r13 = cbrt(rs);
  const double r43 = rs * r13;
  const double x = 0.5 * g / r43;
  const double root = sqrt(1.0 + x * x);
  const double ash = log(x + root);
  const double den = 1.0 + 6.0 * beta * x * ash;
  const double b = x * x / den;
  const double q = x / den;
  const double bp = 2.0 * q - 6.0 * beta * q * q * (ash + x / root);
  GgaTerm t;
  t.f = -2.0 * beta * r43 * b;
  t.dfr = -beta * (4.0 / 3.0) * r13 * (b - x * bp);
  t.dfg = -beta * bp;
  return t;
}

// Lee-Yang-Parr correlation, closed shell (lyp_gcc, cp_becke.C:91-172):
// u = rho^(-1/3), D = 1 + d u, omega = exp(-c u) u^11 / D,
// delta = c u + d u / D, A = C_F rho^(8/3) + (5/12 - 7 delta / 72) g^2 - 11 g^2 / 24,
// f = -a rho / D - a b omega A rho^2.
__device__ __forceinline__ GgaTerm gga_lyp(double rho, double g) {
  const double a = 0.049180, b = 0.1320, c = 0.25330, d = 0.3490;
  const double cf = 2.871234000188191;  // C_F = 0.3 (3 pi^2)^(2/3)
  const double u = 1.0 / cbrt(rho);
  const double u2 = u * u;
  const double den = 1.0 + d * u;
  double u11 = u2 * u2;            // u^4
  u11 = u11 * u11 * u2 * u;        // u^11
  const double om = exp(-c * u) * u11 / den;
  const double dl = c * u + d * u / den;
  const double g2 = g * g;
  const double r2 = rho * rho;
  const double r23i = u2;          // rho^(-2/3)
  const double cq = 5.0 / 12.0 - 7.0 * dl / 72.0;
  const double A = cf * r2 / r23i + cq * g2 - 11.0 * g2 / 24.0;  // C_F rho^(8/3) = C_F rho^2 / rho^(-2/3)
  const double dom = om * (c * u + d * u / den - 11.0) / (3.0 * rho);
  const double ddl = -(u / (3.0 * rho)) * (c + d / (den * den));
  const double dA = (8.0 / 3.0) * cf * rho / r23i - (7.0 / 72.0) * ddl * g2;  // d/drho, rho^(5/3) = rho / rho^(-2/3)
  GgaTerm t;
  t.f = -a * rho / den - a * b * om * A * r2;
  t.dfr = -a * (1.0 + (4.0 / 3.0) * d * u) / (den * den) - a * b * (dom * A * r2 + om * (dA * r2 + 2.0 * A * rho));
  t.dfg = -a * b * om * r2 * 2.0 * g * (cq - 11.0 / 24.0);
  return t;
}

// Per point, on rho > rho_cut = gga_cut / 10 (CP_getGGAFunctional): Becke +
// LYP times the switching function s = t^2 (3 - 2 t), t = clamp((rho -
// rho_cut) / (3.9 gga_cut), 0, 1); vxc += d(s f)/drho; grad <- h; block
// partials of the exchange and correlation parts.  h is 0 where
// |grad rho| = 0 (no direction) and below rho_cut.
__global__ void __launch_bounds__(OA_NTHREADS)
k_rho_gga(const double* __restrict__ rho, double* __restrict__ grad, size_t npts, double gga_cut,
          double* __restrict__ vxc, double* __restrict__ part) {
  __shared__ double sh[2 * 32];
  const double rho_cut = 0.1 * gga_cut, heal = 1.0 / (3.9 * gga_cut);
  double acc[2] = {0.0, 0.0};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < npts; i += (size_t)gridDim.x * blockDim.x) {
    const double r = rho[i];
    double hx = 0.0, hy = 0.0, hz = 0.0;
    if (r > rho_cut) {
      const double gx = grad[i], gy = grad[npts + i], gz = grad[2 * npts + i];
      const double g2 = gx * gx + gy * gy + gz * gz;
      const double g = sqrt(g2);
      const double t = fmin(fmax((r - rho_cut) * heal, 0.0), 1.0);
      const double sw = t * t * (3.0 - 2.0 * t);
      const double dsw = 6.0 * t * (1.0 - t) * heal;
      const GgaTerm x = gga_becke88(r, g), c = gga_lyp(r, g);
      vxc[i] += (x.dfr + c.dfr) * sw + (x.f + c.f) * dsw;
      acc[0] += x.f * sw;
      acc[1] += c.f * sw;
      if (g2 > 0.0) {
        const double k = (x.dfg + c.dfg) * sw / g;
        hx = gx * k; hy = gy * k; hz = gz * k;
      }
    }
    grad[i] = hx;
    grad[npts + i] = hy;
    grad[2 * npts + i] = hz;
  }
  block_sum_n<2>(acc, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x + 0] = acc[0];
    part[2 * blockIdx.x + 1] = acc[1];
  }
}

// g-vector of element (line lb, plane zz) of a z-pass block and whether it
// is inside the density sphere (the points k_rho_zpass keeps, g = 0 out)
__device__ __forceinline__ bool rho_sphere_g(int l, int zz, int ny, int nz, double tpi_l, double ecut4, int ktab,
                                             double* gx, double* gy, double* gz) {
  const int kx = l / ny;
  int ky = l - kx * ny; if (2 * ky >= ny) ky -= ny;
  int kz = zz; if (2 * kz >= nz) kz -= nz;
  *gx = tpi_l * kx; *gy = tpi_l * ky; *gz = tpi_l * kz;
  const double g2 = *gx * *gx + *gy * *gy + *gz * *gz;
  return g2 != 0.0 && g2 <= ecut4 && abs(kx) <= ktab && abs(ky) <= ktab && abs(kz) <= ktab;
}

// z transform of nb lines in x (ld ldz) with y as scratch; returns the
// buffer holding the result
template <int N1, int N2, int SIGN>
__device__ __forceinline__ double2* zfft_any(double2* x, double2* y, int ldz, int nb, const OaFftPlan& pz,
                                             const double2* tw) {
  if constexpr (N1 > 0) {
    zfft2<N1, N2, SIGN>(x, y, ldz, nb, tw);
    return x;
  } else {
    return fft_pingpong<SIGN>(x, y, ldz, nb, pz, tw);
  }
}

// three buffers of OA_LB lines (row stride ldz, each sized for the
// two-pass scratch layout) after the twiddles
template <int N1, int N2>
__host__ __device__ inline int gga_zbuf_ld(int nz) {
  if constexpr (N1 > 0) {
    const int ps = ZLd<N1, N2>::PS;
    return ps > nz + 1 ? ps : nz + 1;
  } else {
    return nz + 1;
  }
}

template <int N1, int N2>
__global__ void __launch_bounds__(OA_NTHREADS, 2)
k_rho_grad_z(const double2* __restrict__ dz, double2* __restrict__ dzg, size_t fstride, int ldl_d, int nlines_d,
             int ny, int nz, OaFftPlan pz, const double2* __restrict__ twz, double tpi_l, double ecut4, int ktab,
             double rvol) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ldz = nz + 1, lb_sz = OA_LB * gga_zbuf_ld<N1, N2>(nz);
  double2* tw = (double2*)smem_raw;
  double2* bufs[3];
  bufs[0] = tw + align_up_r(nz, 2);
  bufs[1] = bufs[0] + lb_sz;
  bufs[2] = bufs[1] + lb_sz;
  const int l0 = blockIdx.x * OA_LB;
  const int nb = min(OA_LB, nlines_d - l0);
  load_twiddles(tw, twz, nz);
  for (int idx = threadIdx.x; idx < nz * OA_LB; idx += blockDim.x) {
    const int zz = idx / OA_LB, lb = idx - zz * OA_LB;
    if (lb < nb) rho_cp16(bufs[0] + lb * ldz + zz, dz + (size_t)zz * ldl_d + l0 + lb);
  }
  rho_cp_commit();
  rho_cp_wait();
  __syncthreads();
  double2* r = zfft_any<N1, N2, -1>(bufs[0], bufs[1], ldz, nb, pz, tw);
  __syncthreads();
  double2* x = (r == bufs[0]) ? bufs[1] : bufs[0];
  double2* y = bufs[2];
  for (int a = 0; a < 3; ++a) {
    for (int idx = threadIdx.x; idx < nb * nz; idx += blockDim.x) {
      const int lb = idx / nz, zz = idx - lb * nz;
      double gx, gy, gz;
      const bool in = rho_sphere_g(l0 + lb, zz, ny, nz, tpi_l, ecut4, ktab, &gx, &gy, &gz);
      const double2 v = r[lb * ldz + zz];
      const double f = in ? (a == 0 ? gx : (a == 1 ? gy : gz)) * rvol : 0.0;
      x[lb * ldz + zz] = make_double2(-v.y * f, v.x * f);  // i g_a rho(g) / V
    }
    __syncthreads();
    double2* q = zfft_any<N1, N2, +1>(x, y, ldz, nb, pz, tw);
    __syncthreads();
    double2* out = dzg + a * fstride;
    for (int idx = threadIdx.x; idx < nz * OA_LB; idx += blockDim.x) {
      const int zz = idx / OA_LB, lb = idx - zz * OA_LB;
      if (lb < nb) out[(size_t)zz * ldl_d + l0 + lb] = q[lb * ldz + zz];
    }
    __syncthreads();
  }
}

template <int N1, int N2>
__global__ void __launch_bounds__(OA_NTHREADS, 2)
k_rho_div_z(double2* __restrict__ dz, const double2* __restrict__ dzh, size_t fstride, int ldl_d, int nlines_d,
            int ny, int nz, OaFftPlan pz, const double2* __restrict__ twz, double tpi_l, double ecut4, int ktab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ldz = nz + 1, lb_sz = OA_LB * gga_zbuf_ld<N1, N2>(nz);
  double2* tw = (double2*)smem_raw;
  double2* a0 = tw + align_up_r(nz, 2);
  double2* a1 = a0 + lb_sz;
  double2* acc = a1 + lb_sz;
  const int l0 = blockIdx.x * OA_LB;
  const int nb = min(OA_LB, nlines_d - l0);
  load_twiddles(tw, twz, nz);
  for (int idx = threadIdx.x; idx < OA_LB * ldz; idx += blockDim.x) acc[idx] = make_double2(0.0, 0.0);
  for (int a = 0; a < 3; ++a) {
    const double2* in = dzh + a * fstride;
    for (int idx = threadIdx.x; idx < nz * OA_LB; idx += blockDim.x) {
      const int zz = idx / OA_LB, lb = idx - zz * OA_LB;
      if (lb < nb) rho_cp16(a0 + lb * ldz + zz, in + (size_t)zz * ldl_d + l0 + lb);
    }
    rho_cp_commit();
    rho_cp_wait();
    __syncthreads();
    const double2* r = zfft_any<N1, N2, -1>(a0, a1, ldz, nb, pz, tw);
    __syncthreads();
    for (int idx = threadIdx.x; idx < nb * nz; idx += blockDim.x) {
      const int lb = idx / nz, zz = idx - lb * nz;
      double gx, gy, gz;
      if (rho_sphere_g(l0 + lb, zz, ny, nz, tpi_l, ecut4, ktab, &gx, &gy, &gz)) {
        const double ga = a == 0 ? gx : (a == 1 ? gy : gz);
        const double2 v = r[lb * ldz + zz];
        acc[lb * ldz + zz].x -= v.y * ga;  // += i g_a h_a(g)
        acc[lb * ldz + zz].y += v.x * ga;
      }
    }
    __syncthreads();
  }
  const double2* q = zfft_any<N1, N2, +1>(acc, a0, ldz, nb, pz, tw);
  __syncthreads();
  for (int idx = threadIdx.x; idx < nz * OA_LB; idx += blockDim.x) {
    const int zz = idx / OA_LB, lb = idx - zz * OA_LB;
    if (lb < nb) {
      double2& o = dz[(size_t)zz * ldl_d + l0 + lb];
      const double2 w = q[lb * ldz + zz];
      o.x -= w.x;
      o.y -= w.y;
    }
  }
}

cudaError_t oa_rho2_fwd(cudaStream_t s, int n, int nz, const double* rho, double scale, const double2* tw,
                        double2* dz, int ldl_d, int nf, size_t fin, size_t fout);
cudaError_t oa_rho_zpass_plain(oa_ctx* c, cudaStream_t s, int nblk, double* part, double* fpart, const EesLocArgs& ees);
cudaError_t oa_rho_zpass_forces(oa_ctx* c, cudaStream_t s, int nblk, double* part, double* fpart,
                                const EesLocArgs& ees);
cudaError_t oa_rho2_bwd(cudaStream_t s, int n, int nz, double2* dz, int ldl_d, const double2* tw,
                        const double* vxc, void* vks, int fp64, int nf, size_t fin, size_t fout);

__global__ void k_phase_tables(const double* __restrict__ pos, int natm, int ktab, double tpi_l, double2* __restrict__ phase) {
  const int nt = 2 * ktab + 1;
  const int total = natm * 3 * nt;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int k = i % nt - ktab;
    const int ax = (i / nt) % 3;
    const int at = i / (3 * nt);
    double sn, cs;
    sincos(tpi_l * (double)k * pos[at * 3 + ax], &sn, &cs);
    phase[i] = make_double2(cs, sn);
  }
}

// ---------------------------------------------------------------------------
size_t oa_rho_plane_smem_bytes(int nx, int ny, int nkx, int npair, int ychunk) {
  return rho_plane_layout(nx, ny, nkx, npair, ychunk).total;
}

// Mixed form: the FP32 transforms scale the density by about 1 - 1.4e-7
// (a uniform gain error); the density is renormalised to the electron count
// of the FP64 coefficients, Q = sum_s occ_s sum_g w |c_sg|^2, against the
// FP32 density's own sum_r rho V/N.  One block, fixed summation order.
__global__ void k_charge_scale(const double* __restrict__ qexact, int n1, const double* __restrict__ q32, int n2,
                               double rnpts, double* __restrict__ scale) {
  __shared__ double sh[2 * 32];
  double v[2] = {0.0, 0.0};
  for (int i = threadIdx.x; i < n1; i += blockDim.x) v[0] += qexact[i];
  for (int i = threadIdx.x; i < n2; i += blockDim.x) v[1] += q32[i];
  block_sum_n<2>(v, sh);
  if (threadIdx.x == 0) scale[0] = (v[1] > 0.0) ? v[0] / (v[1] * rnpts) : 1.0;
}

cudaError_t oa_launch_rho_xc(oa_ctx* c, cudaStream_t s) {
  const int nblk = 4 * 148;
  const bool renorm = c->qvalid == 2;
  if (renorm) {
    k_charge_scale<<<1, 1024, 0, s>>>(c->qpart, c->nq, c->qpart2, c->nq2, 1.0 / (double)c->npts, c->qscale);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  k_rho_xc<<<nblk, OA_NTHREADS, 0, s>>>(c->rho_part, c->rho_ngroup, (size_t)c->npts, 1.0 / c->vol,
                                        c->gga ? 0.0 : 1.0, renorm ? c->qscale : nullptr, c->rho, c->vxc, c->red);
  return cudaGetLastError();
}

int oa_rho_xc_nblk() { return 4 * 148; }
// blocks of the density z pass: sixteen lines with atom forces, else eight
// (RhoZLB)
int oa_rho_z_nblk(const oa_ctx* c) { return c->ions ? (c->nlines_d + 15) / 16 : (c->nlines_d + 7) / 8; }
// offset of the GGA block partials (2 per block of k_rho_gga) in c->red
size_t oa_rho_gga_red_off(const oa_ctx* c) { return (size_t)3 * oa_rho_xc_nblk() + 3 * (size_t)((c->nlines_d + 7) / 8); }

cudaError_t oa_launch_phase_tables(oa_ctx* c, cudaStream_t s) {
  const double tpi_l = 2.0 * 3.14159265358979323846 / c->box;
  const int total = c->natm * 3 * (2 * c->kmax_tab + 1);
  k_phase_tables<<<(total + 255) / 256, 256, 0, s>>>(c->pos, c->natm, c->kmax_tab, tpi_l, c->phase);
  return cudaGetLastError();
}

// x-y forward transform of nf real fields (stride fin doubles) into density
// z-lines (stride fout double2), two-pass kernels where the length has them
static cudaError_t rho_xy_fwd(oa_ctx* c, cudaStream_t s, const double* src, double scale, double2* dst, int nf,
                              size_t fin, size_t fout) {
  cudaError_t e = c->nx == c->ny ? oa_rho2_fwd(s, c->nx, c->nz, src, scale, c->tw_x, dst, c->ldl_d, nf, fin, fout)
                                 : cudaErrorNotSupported;
  if (e != cudaErrorNotSupported) return e;
  RhoPlaneSmem L = rho_plane_layout(c->nx, c->ny, c->nkx_d, c->npair_d, c->ychunk_d);
  e = oa_smem_limit(k_rho_plane_fwd);
  if (e != cudaSuccess) return e;
  k_rho_plane_fwd<<<dim3(c->nz, nf), OA_NTHREADS, L.total, s>>>(src, scale, c->nx, c->ny, c->nz, c->nkx_d,
                                                                 c->plan_x, c->plan_y, c->tw_x, c->tw_y, dst,
                                                                 c->ldl_d, c->npair_d, c->ychunk_d, L, fin, fout);
  return cudaGetLastError();
}

// x-y inverse of nf fields of density z-lines into real grids (+ vxc when
// not null), in FP64 or the compute precision
static cudaError_t rho_xy_bwd(oa_ctx* c, cudaStream_t s, double2* src, const double* vxc, void* dst, int fp64,
                              int nf, size_t fin, size_t fout) {
  cudaError_t e = c->nx == c->ny
                      ? oa_rho2_bwd(s, c->nx, c->nz, src, c->ldl_d, c->tw_x, vxc, dst, fp64, nf, fin, fout)
                      : cudaErrorNotSupported;
  if (e != cudaErrorNotSupported) return e;
  RhoPlaneSmem L = rho_plane_layout(c->nx, c->ny, c->nkx_d, c->npair_d, c->ychunk_d);
  const dim3 grid(c->nz, nf);
  if (fp64) {
    e = oa_smem_limit(k_rho_plane_bwd<double>);
    if (e != cudaSuccess) return e;
    k_rho_plane_bwd<double><<<grid, OA_NTHREADS, L.total, s>>>(src, c->ldl_d, c->nx, c->ny, c->nz, c->nkx_d,
                                                               c->plan_x, c->plan_y, c->tw_x, c->tw_y, vxc,
                                                               (double*)dst, c->npair_d, c->ychunk_d, L, fin, fout);
  } else {
    e = oa_smem_limit(k_rho_plane_bwd<float>);
    if (e != cudaSuccess) return e;
    k_rho_plane_bwd<float><<<grid, OA_NTHREADS, L.total, s>>>(src, c->ldl_d, c->nx, c->ny, c->nz, c->nkx_d,
                                                              c->plan_x, c->plan_y, c->tw_x, c->tw_y, vxc,
                                                              (float*)dst, c->npair_d, c->ychunk_d, L, fin, fout);
  }
  return cudaGetLastError();
}

// the two GGA z kernels, two-pass where nz has a factorisation
static cudaError_t gga_z(oa_ctx* c, cudaStream_t s, int div) {
  const double tpi_l = 2.0 * 3.14159265358979323846 / c->box;
  const size_t fst = (size_t)c->nz * c->ldl_d;
  const int nbz = (c->nlines_d + OA_LB - 1) / OA_LB;
  auto go = [&](auto grad_k, auto div_k, int ld) -> cudaError_t {
    const size_t sm = (align_up_r(c->nz, 2) + (size_t)3 * OA_LB * ld) * sizeof(double2);
    if (sm > (size_t)OA_MAX_SMEM) return cudaErrorNotSupported;
    cudaError_t e2;
    if (div) {
      if ((e2 = oa_smem_limit(div_k)) != cudaSuccess) return e2;
      div_k<<<nbz, OA_NTHREADS, sm, s>>>((double2*)c->dz, (const double2*)c->dzg, fst, c->ldl_d, c->nlines_d, c->ny,
                                         c->nz, c->plan_z, c->tw_z, tpi_l, c->ecut_rho, c->kmax_tab);
    } else {
      if ((e2 = oa_smem_limit(grad_k)) != cudaSuccess) return e2;
      grad_k<<<nbz, OA_NTHREADS, sm, s>>>((const double2*)c->dz, (double2*)c->dzg, fst, c->ldl_d, c->nlines_d,
                                          c->ny, c->nz, c->plan_z, c->tw_z, tpi_l, c->ecut_rho, c->kmax_tab,
                                          1.0 / c->vol);
    }
    return cudaGetLastError();
  };
  cudaError_t e;
  switch (c->nz) {
#define OA_GZ(NN, A, B) \
  case NN: e = go(k_rho_grad_z<A, B>, k_rho_div_z<A, B>, gga_zbuf_ld<A, B>(c->nz)); break;
    OA_LENGTHS_ALL(OA_GZ)
#undef OA_GZ
    default: e = cudaErrorNotSupported; break;
  }
  if (e == cudaErrorNotSupported) e = go(k_rho_grad_z<0, 0>, k_rho_div_z<0, 0>, c->nz + 1);
  return e;
}

// BLYP before the Hartree z pass: grad rho, the per-point functional
// (vxc, EGGA partials, h), and h's x-y forward transform into dzg
static cudaError_t gga_front(oa_ctx* c, cudaStream_t s) {
  const size_t fz = (size_t)c->nz * c->ldl_d, fr = (size_t)c->npts;
  cudaError_t e;
  if ((e = gga_z(c, s, 0)) != cudaSuccess) return e;
  if ((e = rho_xy_bwd(c, s, (double2*)c->dzg, nullptr, c->grad, 1, 3, fz, fr)) != cudaSuccess) return e;
  k_rho_gga<<<oa_rho_xc_nblk(), OA_NTHREADS, 0, s>>>(c->rho, c->grad, fr, c->gga_cut, c->vxc,
                                                      c->red + oa_rho_gga_red_off(c));
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return rho_xy_fwd(c, s, c->grad, 1.0 / c->npts, (double2*)c->dzg, 3, fr, fz);
}

cudaError_t oa_launch_rho_fft_hart(oa_ctx* c, cudaStream_t s) {
  cudaError_t e;
  // phase tables exp(i 2 pi k x / L) (a native step makes them first of all)
  if (!c->phase_done && (e = oa_launch_phase_tables(c, s)) != cudaSuccess) return e;
  if ((e = rho_xy_fwd(c, s, c->rho, c->vol / c->npts, (double2*)c->dz, 1, 0, 0)) != cudaSuccess) return e;
  if (c->gga && (e = gga_front(c, s)) != cudaSuccess) return e;
  const int nbz = oa_rho_z_nblk(c);
  const bool forces = c->ions != nullptr;
  EesLocArgs ees{};
  if (c->eesl) {
    // B-spline grids of the atom types and their transform (and the force
    // grids zeroed) before the z pass reads them
    if ((e = oa_launch_eesl_front(c, s)) != cudaSuccess) return e;
    const oa_eesl* L = c->eesl;
    ees.zq = L->zq;
    ees.zy = forces ? L->zy : nullptr;
    ees.ba = L->ba; ees.bb = L->bb; ees.bc = L->bc;
    ees.gzvps = L->gzvps;
    ees.na = L->na; ees.nb = L->nb; ees.nc = L->nc;
    ees.gstride = (size_t)L->na * L->nb * L->nc;
  }
  double* part = c->red + 3 * oa_rho_xc_nblk();
  e = forces ? oa_rho_zpass_forces(c, s, nbz, part, c->ions->fpart, ees)
             : oa_rho_zpass_plain(c, s, nbz, part, nullptr, ees);
  if (e != cudaSuccess) return e;
  // EES: the force grids back to real space and the atom forces from them
  if (c->eesl && forces && (e = oa_launch_eesl_forces(c, s)) != cudaSuccess) return e;
  // white-byrd: V_KS z-lines -= z^-1 (i g . h(g))
  if (c->gga && (e = gga_z(c, s, 1)) != cudaSuccess) return e;
  return rho_xy_bwd(c, s, (double2*)c->dz, c->vxc, c->vks, c->precision == OA_FP64, 1, 0, 0);
}
