// State-pair plane kernels (oa_pp.cuh): arguments and dispatch over the grid
// lengths.  nx = ny = n.
#pragma once
#include <cuda_runtime.h>

struct PpArgs {
  int mode;              // 0: density pass, 4: V_KS pass, -1: query (dbps, vbps and split only)
  int n;
  cudaStream_t st;
  void* zbuf;
  int nstate, nz, ldl, nlines;
  const int* cols;       // per kx column {first line, ky of the first line, lines, 0}
  int nkx, kymax;
  const double2* tw;
  const double* occ;
  const void* vks;
  double* rho_part;
  int ngroup;
  void* psir;
  double* qpart;         // mode 0, may be null: [group][z][split] sums of occ |psi(r)|^2
  int *dbps, *vbps;      // query: resident blocks per SM of the density and of the V_KS kernel
  int* split;            // query: row splits of the density kernel
};

// cudaErrorNotSupported when the length, the sphere or the shared memory has
// no pair kernel (the callers then use the per-state kernels)
cudaError_t oa_pp_plane(int precision, const PpArgs& A);

struct EesArgs;

struct PeArgs {
  int mode;              // 2: Z gather, 3: scatter, -1: query (bps only)
  int n;
  cudaStream_t st;
  void* zbuf;            // nonlocal-grid z-line buffer
  int nstate, nz, ldl, nlines;
  const int* cols;
  int nkx, kymax;
  const double2* tw;
  int ngroup;
  const EesArgs* E;
  int* bps;
};
// EES nonlocal grid, planes n x n; cudaErrorNotSupported as above
cudaError_t oa_pe_plane(int precision, const PeArgs& A);
