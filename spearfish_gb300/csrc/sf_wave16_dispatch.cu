// Classes and dispatch of the anti-diagonal 16-bit kernel (one translation unit per word count).
#include "sf_internal.cuh"
#include "sf_wave16.h"

namespace sfk {

cudaError_t launch_wave16_4(bool, const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16_6(bool, const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16_8(bool, const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16_10(bool, const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16_12(bool, const AffLaunch&, int, cudaStream_t);

cudaError_t launch_wave16x_4(bool, const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16x_6(bool, const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16x_8(bool, const AffLaunch&, int, cudaStream_t);

cudaError_t launch_wave16c_4(const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16c_6(const AffLaunch&, int, cudaStream_t);
cudaError_t launch_wave16c_8(const AffLaunch&, int, cudaStream_t);

cudaError_t launch_wave16t_4(bool, const AffLaunch&, int, int, cudaStream_t);
cudaError_t launch_wave16xt_4(bool, const AffLaunch&, int, int, cudaStream_t);
cudaError_t launch_wave16xt_8(bool, const AffLaunch&, int, int, cudaStream_t);

// Classes by the cells they hold, within each range.  The cheapest a band cell: a row step costs
// a warp about 32 Q + 60 issue slots whatever it holds, so many cells a lane and many passes a
// warp; Prefix passes keep two more registers a word and stop at 8 words.  The fastest a pass:
// four words a lane, over two to seven warps for bands past 512 cells (two words a lane over up to
// seven warps took as long: a row step's chain through both shuffles is 270 cycles, 400 with
// traceback).
const WaveClass kWave[kWaveN] = {
    {4, 3},  {4, 4},  {6, 3},  {4, 5},  {6, 4},   {10, 3},  {8, 4},   {12, 3},
    {10, 4}, {12, 4}, {10, 5}, {12, 5}, {8, 8},   {12, 6},  {10, 8},  {12, 8},
    {10, 10}, {12, 10}, {8, 16}, {10, 16}, {12, 16}, {8, 32}, {10, 32}, {12, 32},
    {4, 122}, {4, 152}, {4, 182}, {4, 212},
    {4, 8}, {4, 16}, {4, 32}, {4, 62}, {4, 92}, {4, 122}, {4, 152}, {4, 182}, {4, 212},
    {4, 3}, {4, 4}, {6, 3}, {4, 5}, {6, 4}, {8, 4}, {8, 5}, {8, 6}, {8, 8}, {8, 10}, {8, 16}, {8, 32},
    {8, 62}, {8, 92}, {8, 122},
    {4, 8}, {4, 16}, {4, 32}, {4, 62}, {8, 32}, {4, 92}, {4, 122}, {4, 152}, {4, 182}, {4, 212}};

cudaError_t launch_wave16(int q, bool prefix, bool cut, bool team, bool tb, const AffLaunch& a, int grid,
                          int block, cudaStream_t s) {
  if (cut) {
    if (team || tb) return cudaErrorInvalidValue;
    return q == 4   ? launch_wave16c_4(a, grid, s)
           : q == 6 ? launch_wave16c_6(a, grid, s)
           : q == 8 ? launch_wave16c_8(a, grid, s)
                    : cudaErrorInvalidValue;
  }
  if (team) {
    if (q == 4) return (prefix ? launch_wave16xt_4 : launch_wave16t_4)(tb, a, grid, block, s);
    return prefix && q == 8 ? launch_wave16xt_8(tb, a, grid, block, s) : cudaErrorInvalidValue;
  }
  switch (q) {
    case 4: return prefix ? launch_wave16x_4(tb, a, grid, s) : launch_wave16_4(tb, a, grid, s);
    case 6: return prefix ? launch_wave16x_6(tb, a, grid, s) : launch_wave16_6(tb, a, grid, s);
    case 8: return prefix ? launch_wave16x_8(tb, a, grid, s) : launch_wave16_8(tb, a, grid, s);
    case 10: return prefix ? cudaErrorInvalidValue : launch_wave16_10(tb, a, grid, s);
    case 12: return prefix ? cudaErrorInvalidValue : launch_wave16_12(tb, a, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sfk
