// Dispatch of the state-pair plane kernels over precision and length groups.
#include "oa_pp.h"
#include "../../include/oa_gpu.h"

cudaError_t oa_pp_f0(const PpArgs& A);
cudaError_t oa_pp_f1(const PpArgs& A);
cudaError_t oa_pp_f2(const PpArgs& A);
cudaError_t oa_pp_f3(const PpArgs& A);
cudaError_t oa_pp_d0(const PpArgs& A);
cudaError_t oa_pp_d1(const PpArgs& A);
cudaError_t oa_pp_d2(const PpArgs& A);
cudaError_t oa_pp_d3(const PpArgs& A);

cudaError_t oa_pp_plane(int precision, const PpArgs& A) {
  typedef cudaError_t (*Group)(const PpArgs&);
  static const Group mixed[4] = {oa_pp_f0, oa_pp_f1, oa_pp_f2, oa_pp_f3};
  static const Group fp64[4] = {oa_pp_d0, oa_pp_d1, oa_pp_d2, oa_pp_d3};
  for (int k = 0; k < 4; ++k) {
    const cudaError_t e = (precision == OA_FP64 ? fp64 : mixed)[k](A);
    if (e != cudaErrorNotSupported) return e;
  }
  return cudaErrorNotSupported;
}

// the row-pruned EES kernels (oa_pp_ees.cuh)
cudaError_t oa_pe_f(const PeArgs& A);
cudaError_t oa_pe_d(const PeArgs& A);
cudaError_t oa_pe_plane(int precision, const PeArgs& A) { return precision == OA_FP64 ? oa_pe_d(A) : oa_pe_f(A); }
