// shell_lane_rr.cu -- shell_lane_kernel of the ket type RR (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_rr(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_R, SH_R, false, false, false>(db, ncta, st, A);
}
}  // namespace ss
