// Nonlocal-grid pair kernels, FP32.
#include "oa_pp_ees.cuh"
#include "oa_pp_ees_table.h"

cudaError_t oa_pe_f(const PeArgs& A) {
  switch (A.n) {
#define OA_PE_CASE(N, ...) case N: return pe_run<PeCfg<__VA_ARGS__>>(A);
    OA_PE_F(OA_PE_CASE)
#undef OA_PE_CASE
    default: return cudaErrorNotSupported;
  }
}
