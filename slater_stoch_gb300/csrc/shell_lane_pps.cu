// shell_lane_pps.cu -- shell_lane_kernel of the ket type PP, one shell with itself, on one centre (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_pps(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_P, SH_P, true, true, false>(db, ncta, st, A);
}
}  // namespace ss
