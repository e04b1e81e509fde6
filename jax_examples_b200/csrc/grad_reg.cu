// Register-path ERI-derivative adjoint kernels: s and p shells, and the dispatch
// over the classes.
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
  switch (qc) {
    case 6:
    case 7:
    case 8:
    case 9:
      return launch_grad_reg_ds(qc, p, s);
    case 10:
    case 11:
      return launch_grad_reg_dp(qc, p, s);
    case 12:
      return launch_grad_reg_dppp(qc, p, s);
    case 13:
      return launch_grad_reg_dpds(qc, p, s);
    case 14:
      return launch_grad_reg_dpdp(qc, p, s);
    case 15:
    case 16:
      return launch_grad_reg_dd(qc, p, s);
    case 17:
      return launch_grad_reg_ddpp(qc, p, s);
    case 18:
      return launch_grad_reg_ddds(qc, p, s);
    default:
      return launch_grad_reg_sp(qc, p, s);
  }
}

}  // namespace jqc
