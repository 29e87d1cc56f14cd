// Anti-diagonal 16-bit kernels with 8 words a lane and parity, a team of warps a Prefix pass.
#include "sf_wave16_impl.cuh"

namespace sfk {
cudaError_t launch_wave16xt_8(bool tb, const AffLaunch& a, int grid, int block, cudaStream_t s) {
  return launch_wave16t_q<8, true>(tb, a, grid, block, s);
}
}  // namespace sfk
