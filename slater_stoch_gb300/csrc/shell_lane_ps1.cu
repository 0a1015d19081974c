// shell_lane_ps1.cu -- shell_lane_kernel of the ket type PS, on one centre (own translation unit).
#include "shell_lane.cuh"

namespace ss {
cudaError_t launch_lane_ps1(int db, int ncta, cudaStream_t st, const ShArgs& A) {
  return launch_lane_bra<SH_P, SH_S, false, true, false>(db, ncta, st, A);
}
}  // namespace ss
