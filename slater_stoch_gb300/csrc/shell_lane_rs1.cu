// shell_lane_rs1.cu -- shell_lane_kernel of the ket type RS, on one centre (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_rs1(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_R, SH_S, false, true, false>(db, ncta, st, A);
}
}  // namespace ss
