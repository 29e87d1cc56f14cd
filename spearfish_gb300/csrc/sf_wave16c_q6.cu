// Anti-diagonal 16-bit kernels with 6 words a lane and parity, Prefix passes with a cut column.
#include "sf_wave16_impl.cuh"

namespace sfk {
cudaError_t launch_wave16c_6(const AffLaunch& a, int grid, cudaStream_t s) {
  return launch_wave16c_q<6>(a, grid, s);
}
}  // namespace sfk
