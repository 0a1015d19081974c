// shell_lane_rp.cu -- shell_lane_kernel of the ket type RP (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_rp(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_R, SH_P, false, false, false>(db, ncta, st, A);
}
}  // namespace ss
