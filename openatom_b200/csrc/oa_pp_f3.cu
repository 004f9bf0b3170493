// State-pair plane kernels, length group F3 of oa_pp_table.h.
#include "oa_pp.cuh"
#include "oa_pp_table.h"

cudaError_t oa_pp_f3(const PpArgs& A) {
  switch (A.n) {
#define OA_PP_CASE(N, ...) case N: return pp_run<PpCfg<__VA_ARGS__>>(A);
    OA_PP_F3(OA_PP_CASE)
#undef OA_PP_CASE
    default: return cudaErrorNotSupported;
  }
}
