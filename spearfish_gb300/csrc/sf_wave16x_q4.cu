// Anti-diagonal 16-bit kernels with 4 words a lane and parity, Prefix passes.
#include "sf_wave16_impl.cuh"

namespace sfk {
cudaError_t launch_wave16x_4(bool tb, const AffLaunch& a, int grid, cudaStream_t s) {
  return launch_wave16_q<4, true>(tb, a, grid, s);
}
}  // namespace sfk
