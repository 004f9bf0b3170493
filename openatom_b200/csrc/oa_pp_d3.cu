// State-pair plane kernels, length group D3 of oa_pp_table.h.
#include "oa_pp.cuh"
#include "oa_pp_table.h"

cudaError_t oa_pp_d3(const PpArgs& A) {
  switch (A.n) {
#define OA_PP_CASE(N, ...) case N: return pp_run<PpCfg<__VA_ARGS__>>(A);
    OA_PP_D3(OA_PP_CASE)
#undef OA_PP_CASE
    default: return cudaErrorNotSupported;
  }
}
