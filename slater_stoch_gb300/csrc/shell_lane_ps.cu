// shell_lane_ps.cu -- shell_lane_kernel of the ket type PS (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_ps(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_P, SH_S, false, false, false>(db, ncta, st, A);
}
}  // namespace ss
