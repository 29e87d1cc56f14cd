// Anti-diagonal 16-bit kernels with 6 words a lane and parity, Global passes.
#include "sf_wave16_impl.cuh"

namespace sfk {
cudaError_t launch_wave16_6(bool tb, const AffLaunch& a, int grid, cudaStream_t s) {
  return launch_wave16_q<6, false>(tb, a, grid, s);
}
}  // namespace sfk
