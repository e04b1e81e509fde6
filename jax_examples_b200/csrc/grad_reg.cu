// Register-path ERI-derivative adjoint kernels (L <= 4 classes): s and p shells,
// and the dispatch over the bra pair classes.
#include "grad_impl.cuh"

namespace jqc {

cudaError_t launch_grad_reg_sp(int qc, const GradParams& p, cudaStream_t s) {
  switch (qc) {
#define X(Q, A, B, C, D) \
  case Q:                \
    return launch_grad_class<A, B, C, D>(p, s);
    JQC_FOR_GRAD_REG_SP(X)
#undef X
    default:
      return cudaErrorNotSupported;
  }
}

cudaError_t launch_grad_reg(int qc, const GradParams& p, cudaStream_t s) {
  if (!is_grad_reg_class(qc)) return cudaErrorNotSupported;
  switch (qc_bra(qc)) {
    case 3:
      return launch_grad_reg_ds(qc, p, s);
    case 4:
      return launch_grad_reg_dp(qc, p, s);
    case 5:
      return launch_grad_reg_dd(qc, p, s);
    default:
      return launch_grad_reg_sp(qc, p, s);
  }
}

}  // namespace jqc
