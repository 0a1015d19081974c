// shell_k5.cu -- shell_eri_kernel of total degree 5 (own translation unit).
#include "shell_eri.cuh"

namespace ss {
cudaError_t launch_shell_5(int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A) {
  return launch_shell_L<5>(ncta, max_no, max_ni, max_col, st, A);
}
}  // namespace ss
