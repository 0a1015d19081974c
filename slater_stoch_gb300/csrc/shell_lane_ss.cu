// shell_lane_ss.cu -- shell_lane_kernel of the ket type SS (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_ss(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_S, SH_S, false, false, false>(db, ncta, st, A);
}
}  // namespace ss
