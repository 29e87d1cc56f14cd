// Anti-diagonal 16-bit kernels with 4 words a lane and parity, a team of warps a Global pass.
#include "sf_wave16_impl.cuh"

namespace sfk {
cudaError_t launch_wave16t_4(bool tb, const AffLaunch& a, int grid, int block, cudaStream_t s) {
  return launch_wave16t_q<4, false>(tb, a, grid, block, s);
}
}  // namespace sfk
