// Classes of the anti-diagonal 16-bit kernel (sf_wave16_impl.cuh) and what its fields admit,
// shared by the kernel and the plan build.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sfk {

struct AffLaunch;

// Fields: the largest of a pass sits at wave_top after a rebase (each kWaveRebaseRows row
// steps), cells no path reaches at wave_neg; no more than wave_neg is taken off at a rebase or for
// a gap's opening, nor does the largest rise past the field in between.
// The widest Prefix classes leave less at either end.
__host__ __device__ constexpr bool wave_wide(int q, int lanes) { return q * lanes > 256; }
__host__ __device__ constexpr uint32_t wave_top(bool wide) { return wide ? 0xfc00u : 0xf000u; }
__host__ __device__ constexpr uint32_t wave_neg(bool wide) { return wide ? 0x400u : 0x1000u; }
constexpr int kWaveRebaseRows = 32;

// A class: Q words (2Q band cells) a lane and parity, L lanes a pass, 32 / L passes a warp;
// it holds bands of up to 4 Q L cells.
struct WaveClass {
  int q, lanes;
};
extern const WaveClass kWave[];
// Global passes: [0, kWaveFast) the cheapest a cell, [kWaveFast, kWaveX) the fastest a pass;
// Prefix passes: [kWaveX, kWaveXFast) and [kWaveXFast, kWaveN) likewise.
constexpr int kWaveFast = 28, kWaveX = 37, kWaveXFast = 52, kWaveN = 62;
// More than 32 lanes: a team of warps, 30 lanes further on each.
inline int wave_warps(const WaveClass& c) { return c.lanes > 32 ? (c.lanes - 2) / 30 : 1; }
inline int wave_cap(const WaveClass& c) { return 4 * c.q * c.lanes; }
// Traceback words of a pass of `steps` row steps: 2Q words a lane and group of four.
inline uint64_t wave_tb_words(const WaveClass& c, uint64_t steps) {
  return (steps + 3) / 4 * 2 * (uint64_t)c.q * (uint64_t)c.lanes;
}

// A team's warps at most, and the blocks of that many per SM its registers are held to.
__host__ __device__ constexpr int wave_most_warps(int q) { return q <= 4 ? 7 : 4; }
__host__ __device__ constexpr int wave_team_blocks(int q, bool tb, bool ext) {
  return q > 4 ? 3 : ext ? 2 : tb ? 3 : 4;
}
// 4-warp blocks per SM the registers are held to: as many as cost no spill or reload of constants
// (600 2 kb windows, four words: 1.00 ms at five blocks, 0.82 at four; 20,000 Global pairs, ten
// and twelve words: 5.19 ms at three, 5.09 at four; without traceback 600 pairs, four words:
// 0.312 ms at eight, 0.238 at five, and 10,000 of eight words 1.08 at six, 1.05 at five).
__host__ __device__ constexpr int wave_blocks(int q, bool tb, bool ext) {
  return ext ? (tb ? (q <= 6 ? 4 : 3) : 4)
             : tb ? (q <= 4 ? 6 : q <= 6 ? 5 : 4) : (q <= 8 ? 5 : 4);
}

// prefix: Prefix passes, else Global ones; cut: with a cut column (no teams, no traceback).
// block: 128, or a team's threads.
cudaError_t launch_wave16(int q, bool prefix, bool cut, bool team, bool tb, const AffLaunch& a, int grid,
                          int block, cudaStream_t s);

}  // namespace sfk
