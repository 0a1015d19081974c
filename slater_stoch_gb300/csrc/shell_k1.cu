// shell_k1.cu -- shell_eri_kernel of total degree 1 (own translation unit).
#include "shell_eri.cuh"

namespace ss {
cudaError_t launch_shell_1(int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A) {
  return launch_shell_L<1>(ncta, max_no, max_ni, max_col, st, A);
}
}  // namespace ss
