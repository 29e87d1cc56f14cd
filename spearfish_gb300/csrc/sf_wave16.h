// Classes of the anti-diagonal 16-bit kernel (sf_wave16_impl.cuh) and what its fields admit,
// shared by the kernel and the plan build.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sfk {

struct AffLaunch;

// Fields: the largest of a pass sits at kWaveTop after a rebase (each kWaveRebaseRows row
// steps), cells no path reaches at kWaveNeg; no more than kWaveNeg is taken off at a rebase, nor
// does the largest rise past the field in between.
constexpr uint32_t kWaveTop = 0xf000u, kWaveNeg = 0x1000u;
constexpr int kWaveRebaseRows = 32;

// A class: Q words (2Q band cells) a lane and parity, L lanes a pass, 32 / L passes a warp;
// it holds bands of up to 4 Q L cells.
struct WaveClass {
  int q, lanes;
};
extern const WaveClass kWave[];
// Global passes: [0, kWaveFast) the cheapest a cell, [kWaveFast, kWaveX) the fastest a pass;
// Prefix passes: [kWaveX, kWaveXFast) and [kWaveXFast, kWaveN) likewise.
constexpr int kWaveFast = 24, kWaveX = 30, kWaveXFast = 42, kWaveN = 47;
// More than 32 lanes: a team of warps, 30 lanes further on each.
inline int wave_warps(const WaveClass& c) { return c.lanes > 32 ? (c.lanes - 2) / 30 : 1; }
inline int wave_cap(const WaveClass& c) { return 4 * c.q * c.lanes; }
// Traceback words of a pass of `steps` row steps: 2Q words a lane and group of four.
inline uint64_t wave_tb_words(const WaveClass& c, uint64_t steps) {
  return (steps + 3) / 4 * 2 * (uint64_t)c.q * (uint64_t)c.lanes;
}

// 4-warp blocks per SM the registers are held to.
__host__ __device__ constexpr int wave_blocks(int q, bool tb, bool ext) {
  return ext ? (tb ? (q <= 4 ? 5 : q <= 6 ? 4 : 3) : (q <= 4 ? 6 : q <= 6 ? 5 : 4))
             : tb ? (q <= 4 ? 6 : q <= 6 ? 5 : q <= 8 ? 4 : 3) : (q <= 6 ? 8 : q <= 8 ? 6 : q <= 10 ? 5 : 4);
}

// prefix: Prefix passes, else Global ones.  block: 128, or a team's threads.
cudaError_t launch_wave16(int q, bool prefix, bool team, bool tb, const AffLaunch& a, int grid,
                          int block, cudaStream_t s);

}  // namespace sfk
