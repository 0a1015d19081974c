// shell_k6.cu -- shell_eri_kernel of total degree 6 (own translation unit).
#include "shell_eri.cuh"

namespace ss {
cudaError_t launch_shell_6(int ncta, int max_no, int max_ni, int max_col, cudaStream_t st, const ShArgs& A) {
  return launch_shell_L<6>(ncta, max_no, max_ni, max_col, st, A);
}
}  // namespace ss
