// shell_lane_ds1.cu -- shell_lane_kernel of the ket type DS, on one centre (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_ds1(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_D, SH_S, false, true, false>(db, ncta, st, A);
}
}  // namespace ss
