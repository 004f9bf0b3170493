// Density z pass without atom forces (oa_rho_zpass.cuh).
#include "oa_rho_zpass.cuh"

cudaError_t oa_rho_zpass_plain(oa_ctx* c, cudaStream_t s, int nblk, double* part, double* fpart, const EesLocArgs& ees) {
  return rho_zpass<false>(c, s, nblk, part, fpart, ees);
}
