// shell_lane_pp.cu -- shell_lane_kernel of the ket type PP (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_pp(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_P, SH_P, false, false, false>(db, ncta, st, A);
}
}  // namespace ss
