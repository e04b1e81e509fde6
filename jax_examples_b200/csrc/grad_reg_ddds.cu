// Register-path ERI-derivative adjoint kernels: (dd|ds).
#include "grad_impl.cuh"

namespace jqc {

cudaError_t launch_grad_reg_ddds(int qc, const GradParams& p, cudaStream_t s) {
  switch (qc) {
#define X(Q, A, B, C, D) \
  case Q:                \
    return launch_grad_class<A, B, C, D>(p, s);
    JQC_FOR_GRAD_REG_DDDS(X)
#undef X
    default:
      return cudaErrorNotSupported;
  }
}

}  // namespace jqc
