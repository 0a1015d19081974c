// shell_lane_rs4.cu -- shell_lane_kernel of the ket type RS, all four shells on one centre (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_rs4(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_R, SH_S, false, true, true>(db, ncta, st, A);
}
}  // namespace ss
