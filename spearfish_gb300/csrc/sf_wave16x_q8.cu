// Anti-diagonal 16-bit kernels with 8 words a lane and parity, Prefix passes.
#include "sf_wave16_impl.cuh"

namespace sfk {
cudaError_t launch_wave16x_8(bool tb, const AffLaunch& a, int grid, cudaStream_t s) {
  return launch_wave16_q<8, true>(tb, a, grid, s);
}
}  // namespace sfk
