// Global and Prefix banded affine (Gotoh) passes swept by anti-diagonals, two cells per 32-bit
// register and several passes per warp (align.rs:2446-2666 `run_core` in Mode::Global without
// clip or cut, and in Mode::Prefix with or without clip and cut).  Results and traceback
// decisions equal the row kernels' (sf_affine16_impl.cuh).
//
// Cells.  Band offset K = j - i + bl of cell (i, j) sits at a fixed place: lane K / 4Q of the
// pass's L lanes, and along anti-diagonal i + j = t the cells of one parity of K are computed
// together, each from its neighbours K - 1 (left), K + 1 (above) and its own last value (the
// diagonal).  No cell of a step depends on another, so a step has no scan and no serial chain:
// two neighbour shuffles, then 2Q independent cells a lane.  A row step a is one even and one
// odd step; cell K = 2k (+1) is then row i = a - k, column j = a + k - bl (+1).
//
// Fields.  A 16-bit field holds 4 * (value + ext * (i + j)) + offset: the potential makes gap
// extension free, so E = max(Hleft - open, Eleft) and F = max(Hup - open, Fup) are one
// two-operand maximum each (the subtraction is an IMAD, off the pipe the maxima use), and with
// mis = 2 * ext a mismatch adds 0.  The factor 4 leaves two low bits for the traceback: the
// diagonal carries 2, F 1, E 0, so that one three-way maximum also says which won, ties in the
// walk's order (diagonal, F, E); an opened gap carries 2 against an extended one's 0 (E) or 1
// (F), so that a tie opens.  Per cell and row four bits are kept: (winner << 2) | (E opened
// << 1) | F extended.
//
// Band edges.  Left of the band lane 0 takes NEG from outside.  Right of it (and at K = 0 when
// `below` is even, which keeps bl odd) pad cells are computed with every match masked.  A path
// through them leaves the band and returns by gaps and mismatches only, so it costs at least
// 2 * open + 2 * ext * d for the d diagonals it gains, where the band's edge offers d mismatches
// at 2 * ext each: with open >= 1 it never reaches a band cell's maximum, and where an extended
// gap ties an opened one the opened one wins, as in the row kernels.  Cells before row 1 or
// column 1 are masked too, so row 0 and column 0 come out of the recurrence itself, from the
// one seed at (0, 0).  Cells past the text or pattern hold values nothing in the matrix reads.
//
// Prefix passes (EXT) need each row's largest value and its leftmost column, in row order: for
// the clip score, its cell and the X-drop stop, and for the last row's score.  Both travel along
// the row from left to right, an even and the odd cell after it a row step, M = max(M, H even,
// H odd) with the leftmost offset it was reached at, and leave the band at its last cell, where
// one lane keeps the pass's books in row order, four rows at a time.  The rows that run ahead of
// a stop are computed and left out.  Columns past the text count for nothing (the last rows).
// With a cut column (CUT) a second maximum, over the cells up to it, travels beside M.
// 8,000 2 kb windows (band 128, CIGARs) on GB300: row kernel 8.75 ms, a cell a step with its books
// a row at a time 5.95, now 4.83; without CIGARs 7.2 -> 2.94.
//
// Bound: the ALU pipe (one instruction every other cycle a scheduler): 8.5 of a word's 14.5
// instructions with traceback, 4.5 of 6.5 without.  With 12 words a lane and 6 lanes a pass a
// row step issues 459 instructions for five 2 kb passes of band 128 (266 on the ALU pipe, 73% of
// its rate), the row kernel 254 for one; score only 221 (87%) against 150.  20,000 such pairs on
// GB300: 10.25 -> 4.8 ms with CIGARs, 5.7 -> 2.4 ms without.
#pragma once
#include <type_traits>

#include "sf_affine_impl.cuh"
#include "sf_wave16.h"

namespace {

constexpr uint32_t kW2 = 0x00010001u;
constexpr int kWRebase = sfk::kWaveRebaseRows;

// The 16 two-bit fields of x in reverse order.
__device__ __forceinline__ uint32_t rev2(uint32_t x) {
  const uint32_t y = __brev(x);
  return ((y >> 1) & 0x55555555u) | ((y & 0x55555555u) << 1);
}

// Bit 2e set for e < c (register r of the mask: e = 16r ..).
__device__ __forceinline__ uint32_t low_fields(int32_t c, int r) {
  const int32_t k = min(max(c - 16 * r, 0), 16);
  return (uint32_t)((uint64_t(1) << (2 * k)) - 1u) & 0x55555555u;
}

// x * I + y on the multiply-add pipe, whatever I is: the maxima need the other one.
template <int I>
__device__ __forceinline__ uint32_t mad(uint32_t x, uint32_t y) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "n"(I), "r"(y));
  return d;
}
// (x & m) | o in one instruction.
__device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t m, uint32_t o) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(x), "r"(m), "r"(o));
  return d;
}
// x's bits where m is set, y's elsewhere.
__device__ __forceinline__ uint32_t pick(uint32_t x, uint32_t y, uint32_t m) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(d) : "r"(x), "r"(y), "r"(m));
  return d;
}

// Walks the warp's paths from their end cells, each by its pass's lanes, side by side.  Lane d of
// a pass caches eight band offsets (two quads of four) of the row steps 8 (H0 - d) .. + 7, eight
// nibbles an offset, latest row first; a run of diagonal steps, which keeps its band offset, is
// found by one ballot over the cached nibbles.  `steps`: the lane's pass's row steps.
//
// A stored word holds its four row steps' nibbles, each 8 low, on top of the word of the four
// steps before, 16 bits up (the rows push and never clear): its low field needs 0x8888 added, its
// high field that and the earlier word's low field taken off.
//
// L: the lanes of the layout; WL of them (a team: its first warp's) walk.
template <int Q>
__device__ void walk_wave(const sfk::AffLaunch& a, uint32_t jid, bool has, int L, int WL, int l,
                          int base, int32_t steps) {
  const DJob J = a.jobs[jid];
  const TJob T = a.tjobs[jid];
  const DRes R = a.out[jid];
  const int32_t m = (int32_t)J.m, n = (int32_t)J.n;
  const int32_t bl = clamp30(J.below) | 1, W = bl + clamp30(J.above) + 1;
  const int32_t a1 = (bl >> 1) + 1;  // the row step that row-step index 0 stands for
  const int32_t gstride = (Q / 2) * L, groups = (steps + 3) >> 2;  // uint4s per group of four steps
  const uint4* tb = reinterpret_cast<const uint4*>(a.tb + J.tb_word);
  const uint32_t lanes = WL == 32 ? FULL : (1u << WL) - 1u;
  uint32_t* out = a.ops + T.ops_off;
  const uint32_t cap = T.ops_cap;
  uint32_t n_ops = 0, cur_op = 15, cur_len = 0;
  int status = 0;
  // End cell (align.rs:2643-2650 score_col; 975-981 the window's choice).
  int32_t score = R.score, i = m, j = (int32_t)R.score_col;
  if (T.kind != 0) {
    score = sat_add(R.score, T.end_bonus);
    if (R.clip_best >= score) {
      score = R.clip_best;
      i = (int32_t)R.clip_i;
      j = (int32_t)R.clip_j;
      cur_op = 4;
      cur_len = (uint32_t)(m - i);
    }
  }
  const int32_t ei = i, ej = j;
  int32_t K = j - i + bl;
  int state = 0;              // 0 H, 1 E, 2 F
  int32_t H0 = -1, q0 = -1;   // cached: row steps up to 8 H0 + 7, offsets 4 q0 .. 4 q0 + 7
  uint32_t c[8];
#pragma unroll
  for (int x = 0; x < 8; ++x) c[x] = 0;
  // One quad of four offsets in the two groups of row steps 8 h ..: the low or the high fields of
  // its four words, the later group's in the low half.
  auto quad = [&](int32_t h, int32_t kq, uint32_t (&w)[4]) {
    uint4 g[3] = {};  // groups 2 h - 1 (for the high fields), 2 h, 2 h + 1
    uint32_t s = 0x5410u;
    if (h >= 0 && kq >= 0 && kq < Q * L) {
      const int32_t ln = kq / Q, rem = kq - ln * Q, hi = rem >= Q / 2;
      const uint4* p = tb + (rem - (hi ? Q / 2 : 0)) * L + ln;
      if (hi) s = 0x7632u;
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const int32_t k = 2 * h - 1 + u;
        if ((u > 0 || hi) && k >= 0 && k < groups) g[u] = p[(int64_t)k * gstride];
      }
    }
    auto both = [&](uint32_t x0, uint32_t x1, uint32_t x2) {
      return __byte_perm(x2 - (x1 << 16) + 0x88888888u, x1 - (x0 << 16) + 0x88888888u, s);
    };
    w[0] = both(g[0].x, g[1].x, g[2].x);
    w[1] = both(g[0].y, g[1].y, g[2].y);
    w[2] = both(g[0].z, g[1].z, g[2].z);
    w[3] = both(g[0].w, g[1].w, g[2].w);
  };
  const int64_t guard = 3 * ((int64_t)m + n) + 64;
  bool done = !has;
  for (int64_t it = 0; __any_sync(FULL, !done); ++it) {
    const bool end = !done && state == 0 && (i == 0 || j == 0);
    const bool bad = !done && !end && (i <= 0 || j <= 0 || K < 0 || K >= W || it > guard);
    const bool go = !done && !end && !bad;
    const int32_t rho = i + (K >> 1) - a1, h = rho >> 3, pos = 7 - (rho & 7);
    if (go && (K < 4 * q0 || K >= 4 * q0 + 8 || q0 < 0 || h > H0 || h <= H0 - WL)) {
      q0 = max(K - 2, 0) >> 2;
      H0 = h;
      uint32_t w0[4], w1[4];
      quad(h - l, q0, w0);
      quad(h - l, q0 + 1, w1);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        c[x] = w0[x];
        c[4 + x] = w1[x];
      }
    }
    const int32_t x = K - 4 * q0;  // 0 .. 7
    const uint32_t x0 = x & 1 ? c[1] : c[0], x1 = x & 1 ? c[3] : c[2], x2 = x & 1 ? c[5] : c[4],
                   x3 = x & 1 ? c[7] : c[6];
    const uint32_t y0 = x & 2 ? x1 : x0, y1 = x & 2 ? x3 : x2;
    const uint32_t v = x & 4 ? y1 : y0;  // this lane's eight nibbles at K
    const int32_t d = go ? H0 - h : 0;
    const uint32_t nib = (__shfl_sync(FULL, v, min(base + d, 31)) >> (4 * pos)) & 15u;
    // Diagonal cells; rows after the path's own count as such.
    uint32_t nd = ~((v >> 3) & ~(v >> 2)) & 0x11111111u;
    if (l == d) nd &= ~((1u << (4 * pos)) - 1u);
    const uint32_t part = nd ? (uint32_t)(__ffs((int)nd) - 1) >> 2 : 8u;
    const uint32_t nf = ((__ballot_sync(FULL, nd != 0) >> base) & lanes) >> d;
    const int32_t z = nf ? __ffs((int)nf) - 1 : WL - d;  // whole lanes from lane d on
    const int32_t tail = (int32_t)__shfl_sync(FULL, part, min(base + d + z, 31));
    uint32_t op = 0, len = 0;
    if (end) {
      op = i == 0 ? 2 : 1;
      len = (uint32_t)(i == 0 ? j : i);
    }
    if (go) {
      if (state == 0) {
        const uint32_t win = nib >> 2;
        if (win == 2u) {
          const int32_t run = min(8 * z - pos + (nf ? tail : 0), min(i, j));
          len = (uint32_t)run;
          i -= run;
          j -= run;
        } else {
          state = win == 1u ? 2 : 1;
        }
      }
      if (state == 1) {
        op = 2;
        len = 1;
        state = (nib & 2u) ? 0 : 1;
        --j;
        --K;
      } else if (state == 2) {
        op = 1;
        len = 1;
        state = (nib & 1u) ? 2 : 0;
        --i;
        ++K;
      }
    }
    if (len) {
      if (op == cur_op) {
        cur_len += len;
      } else {
        if (cur_len) {
          if (n_ops == cap)
            status = -1;
          else if (l == 0)
            out[n_ops] = (cur_len << 4) | cur_op;
          ++n_ops;
        }
        cur_op = op;
        cur_len = len;
      }
    }
    if (bad) status = 1;
    done = done || end || bad || status != 0;
  }
  if (has && l == 0) {
    if (!status && cur_len) {
      if (n_ops == cap)
        status = -1;
      else
        out[n_ops] = (cur_len << 4) | cur_op;
      ++n_ops;
    }
    TRes tr;
    tr.score = score;
    tr.status = status;
    tr.end_i = (uint32_t)ei;
    tr.end_j = (uint32_t)ej;
    tr.text_start = 0;
    tr.n_ops = status == 0 ? n_ops : 0;
    a.tres[jid] = tr;
  }
}

// A team's exchanges, by turns: each warp's lane 30 for the next warp's lane 0, its lane 1 for the
// last warp's lane 31, its largest field, and whether the pass has ended.
template <int Q, bool EXT>
struct WaveTeam {
  static constexpr int kWarps = sfk::wave_most_warps(Q);
  uint4 up[2][kWarps][Q], down[2][kWarps][Q];
  uint2 row[EXT ? 2 : 1][EXT ? kWarps : 1][Q];
  uint32_t top[2][kWarps];
  uint32_t ended[2];
  uint32_t task;
};

// A Prefix pass's books, in fields' units (four to one), without the potential, kept off the registers.  A
// row's maximum is in the potential of offset 2 kw + 1 (an odd last cell: + 2): pot4 at row 0, row4
// a row.  best (at row i, offset k): the largest so far; a row more than xd below it ends the pass.
struct WaveBooks {
  int32_t best, i, k, clip, xd, pot4, row4, row0, m, tail, at;
  int32_t cut, cut_row, cut_tail;  // CUT: the largest up to the cut, and the last rows it matters for
};
// Prefix passes: the words of the lane that holds a band's last cell over four row steps, by the
// pass's place in its warp, for that lane to pick one by its offset (a select over registers
// costs the ALU pipe 4 Q a row step), and the books.
template <int Q, bool EXT>
struct WaveLast {
  static constexpr int kQuads = EXT ? (Q + 3) / 4 : 1, kSlots = EXT ? 11 : 1;
  uint4 w[kSlots][4][4][kQuads];  // the last slot takes what the other lanes write
  WaveBooks books[kSlots];
};

// One warp's passes, one per segment of L lanes: `jid` is the lane's own pass (any valid one
// where `has` is false: computed, not stored).  TEAM: one pass over the block's warps, 30 lanes
// further on each; a warp's outer lanes (but the first's first and the last's last) repeat its
// neighbours' and are set right from them every 2Q row steps, which is as long as what they lack
// at their outer side takes to cross them, a cell a step.
template <int Q, bool TB, bool EXT, bool TEAM, bool CUT>
__device__ __forceinline__ void wave_passes(const sfk::AffLaunch& a, uint32_t jid, bool has, int L,
                                            int lane, int seg, WaveLast<Q, EXT>& Z,
                                            WaveTeam<Q, EXT>* X) {
  const bool wide = TEAM && EXT && sfk::wave_wide(Q, L);
  const uint32_t kWTop = sfk::wave_top(wide), kWNeg = sfk::wave_neg(wide);
  constexpr int NT = (2 * Q + 15) / 16;  // 16-base registers of a lane's text (pattern) window
  constexpr int NC = (Q + 7) / 8;        // registers of a step's match bits
  static_assert(Q % 2 == 0 && Q >= 4 && Q <= 16, "words per lane and parity");
  const int w = TEAM ? threadIdx.x >> 5 : 0, NW = TEAM ? blockDim.x >> 5 : 1;
  const int l = TEAM ? 30 * w + lane : lane - seg * L;
  const bool leftmost = TEAM ? lane == 0 : l == 0, rightmost = TEAM ? lane == 31 : l == L - 1;
  const bool own = !TEAM || ((lane > 0 || w == 0) && (lane < 31 || w == NW - 1));
  const DJob J = a.jobs[jid];
  const DParams S = a.params[jid];
  const int32_t m = (int32_t)J.m, n = (int32_t)J.n;
  const int32_t below = clamp30(J.below), above = clamp30(J.above);
  const int32_t bl = below | 1, W = bl + above + 1;
  const int32_t k0 = 2 * Q * l;  // the lane's first pair of offsets
  const int32_t a1 = (bl >> 1) + 1;
  // Row steps until cell (m, n) is done; EXT: until row m's last band cell is.
  const int32_t kw = (W - 1) >> 1;  // the pair of offsets the band's last cell is in
  const int32_t N = EXT ? m + kw - a1 + 1 : (m + n + 1) >> 1;

  // The tag masks, opaque so that each use is one three-input instruction.
  const uint32_t one = (uint32_t)opaque_one();
  const uint32_t mlow = 0xfffcfffcu * one, kone = kW2 * one, ktwo = 2u * kone, msel = ~kone;
  const uint32_t mg2 = 0u - 4u * (uint32_t)S.open * kW2;
  const uint32_t v1 = (uint32_t)(S.mat + S.mis), v4 = 4u * v1;
  constexpr uint32_t kH = TB ? 2u : 0u, kF = TB ? 1u : 0u;  // a clean field's low bits
  const uint32_t kNegH = (kWNeg + kH) * kW2, kNegE = kWNeg * kW2, kNegF = (kWNeg + kF) * kW2, kNegM = (kWNeg + 2u) * kW2;

  // EXT: M's potential rises by 4 ext a step, so the top leaves room for a row's width of them.
  const int32_t wtop = EXT ? (int32_t)kWTop - 4 * S.ext * (W + 1) : (int32_t)kWTop;
  [[maybe_unused]] const int32_t cut =
      CUT ? (int32_t)(J.cut < (uint64_t)n + 1 ? J.cut : (uint64_t)n + 1) : 0;
  uint32_t HA[Q], HB[Q], E[Q], F[Q], acc[TB ? 2 * Q : 1];
  uint32_t M[EXT ? Q : 1], MK[EXT ? Q : 1];  // a row's largest value so far and its offset K
  uint32_t C[CUT ? Q : 1];                   // the same up to the cut column
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    // The seed at (0, 0): offset bl, odd.
    const int32_t e = (bl >> 1) - k0;
    const uint32_t top = (uint32_t)wtop + kH, neg = kWNeg + kH;
    HA[k] = kNegH;
    HB[k] = (e == k ? top : neg) | ((e == Q + k ? top : neg) << 16);
    E[k] = kNegE;
    F[k] = kNegF;
    if constexpr (TB) acc[2 * k] = acc[2 * k + 1] = 0;
    if constexpr (EXT) {
      M[k] = kNegM;
      MK[k] = 0;
    }
    if constexpr (CUT) C[k] = kNegM;
  }
  int32_t off = -wtop;

  // Windows: T[r] holds the text bases of columns from a + k0 - bl + 16 r on (T[NT]: the bases
  // that shift in next), P[r] the pattern bases of rows from a - k0 - 16 r downwards, Pn the
  // ones that come next, first at the top.  Both move by one base a row step.
  const int32_t tlim = (n >> 4) + 64, plim = (m >> 4) + 64;  // the pool's slack covers 100 words
  auto word = [&](uint64_t w, int32_t x, int32_t lim) {
    return __ldg(a.pool + w + (uint32_t)min(max(x, 0), lim));
  };
  auto chunk = [&](uint64_t w, int32_t x, int32_t lim) {
    return __funnelshift_r(word(w, x >> 4, lim), word(w, (x >> 4) + 1, lim), 2 * (x & 15));
  };
  uint32_t T[NT + 1], P[NT], Pn;
  const int32_t tx = a1 + k0 - bl, px = a1 - k0;  // at row-step index 0
#pragma unroll
  for (int r = 0; r <= NT; ++r) T[r] = chunk(J.t_word, tx + 16 * r, tlim);
#pragma unroll
  for (int r = 0; r < NT; ++r) P[r] = rev2(chunk(J.p_word, px - 16 * r - 15, plim));
  Pn = rev2(chunk(J.p_word, px + 1, plim));
  uint32_t t0 = 0, t1 = 0, p0 = 0, p1 = 0;  // the next chunk's words, loaded 16 row steps ahead
  const int32_t tsh = 2 * (tx & 15), psh = 2 * ((px + 1) & 15);

  uint32_t Me[NT], Mo[NT];  // match masks of the even and odd step
  // Cells of row step index r that lie in the matrix and the band.
  auto masks = [&](int32_t r) {
    const int32_t x = a1 + r;
    const int32_t rows = x - k0;  // e < rows: row 1 or later
    const int32_t lo_e = max(bl + 1 - x - k0, l == 0 ? bl - below : 0);
    const int32_t lo_o = bl - x - k0;
    const int32_t hi_e = min(rows, ((W + 1) >> 1) - k0), hi_o = min(rows, (W >> 1) - k0);
#pragma unroll
    for (int r2 = 0; r2 < NT; ++r2) {
      Me[r2] = low_fields(min(hi_e, 2 * Q), r2) & ~low_fields(lo_e, r2);
      Mo[r2] = low_fields(min(hi_o, 2 * Q), r2) & ~low_fields(lo_o, r2);
    }
  };
  // Row steps after which every cell of the band is in the matrix (masks constant).
  int32_t rF = max(min(2 * Q * L, (W >> 1) + 1), bl + 1) - a1;
  int32_t Rtot = has ? N : 0;
  rF = __reduce_max_sync(FULL, rF);
  Rtot = (__reduce_max_sync(FULL, Rtot) + 3) & ~3;
  int32_t next_end = __reduce_min_sync(FULL, has ? N : INT32_MAX);

  // A step's match bits: cell k's low field at bit 2 (k % 8) of register k / 8, its high field
  // (cell k + Q) 16 bits up.
  auto matches = [&](const uint32_t (&M)[NT], uint32_t (&cb)[NC]) {
    uint32_t eq[NT];
#pragma unroll
    for (int r = 0; r < NT; ++r) {
      const uint32_t x = T[r] ^ P[r];
      eq[r] = ~(x | (x >> 1)) & M[r];
    }
    if constexpr (Q == 8) {
      cb[0] = eq[0];
    } else if constexpr (Q < 8) {
      cb[0] = __byte_perm(eq[0], eq[0] << (16 - 2 * Q), 0x7610);
    } else {
      const uint32_t hi = Q == 16 ? eq[1] : __funnelshift_r(eq[0], eq[1], 2 * Q);
      cb[0] = __byte_perm(eq[0], hi, 0x5410);
      cb[NC - 1] = __byte_perm(eq[0], hi, 0x7632);
    }
  };
  // EXT: a row's largest value, left to right a pair of offsets (an even and an odd cell, both of
  // one row step) at a time.  It is kept a pair ahead (8 ext more) with bit 1 set, which no cell
  // has there, so that a tie keeps the left one and bit 1 says which won; an even cell has bit 0
  // set, which then stands for the parity of the maximum's offset.  MK: the pair's even offset.
  const uint32_t e4 = 4u * (uint32_t)S.ext * kW2;
  const uint32_t ha = e4 + (TB ? ~0u * kW2 : kW2), hb = 0u - 2u * kW2;  // cells' low bits: kH
  const uint32_t m8 = 2u * e4 + 2u * kW2, kc0 = 4u * (uint32_t)Q * (uint32_t)l * kW2;
  auto row_max = [&](uint32_t xa, uint32_t xb, uint32_t kc, uint32_t ml, uint32_t pl, uint32_t& mo,
                     uint32_t& po) {
    const uint32_t x = __vimax3_u16x2(ml, xa, xb);
    const uint32_t kept = x & (2u * kW2);
    po = pick(pl, kc, mad<0x7fff>(kept, 0u));
    mo = mad<-1>(kept, mad<1>(x, m8));
  };
  // The band's last cell: one lane's word and half, in the even or the odd step.
  const bool last_odd = (W - 1) & 1;
  const int32_t last_e = kw - k0;  // 0 .. 2Q - 1 in the lane that holds it
  const bool books = EXT && has && own && last_e >= 0 && last_e < 2 * Q;
  const bool any_even = EXT && __any_sync(FULL, books && !last_odd);
  const bool any_odd = EXT && __any_sync(FULL, books && last_odd);
  const uint32_t pad0 = l == 0 && bl != below ? 0xffff0000u : ~0u;  // offset 0 is a pad
  constexpr int kSpare = WaveLast<Q, EXT>::kSlots - 1, kArray = 8 * WaveLast<Q, EXT>::kQuads;
  auto* const last = Z.w[books ? seg : kSpare];
  auto* const even_last = Z.w[books && !last_odd ? seg : kSpare];
  auto* const odd_last = Z.w[books && last_odd ? seg : kSpare];
  auto put_last = [&](uint4* to, const uint32_t (&x)[EXT ? Q : 1]) {
    if constexpr (EXT) {
#pragma unroll
      for (int q = 0; q < Q / 4; ++q)
        to[q] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
      if constexpr (Q % 4 != 0) *reinterpret_cast<uint2*>(to + Q / 4) = make_uint2(x[Q - 2], x[Q - 1]);
    }
  };
  volatile WaveBooks& bk = Z.books[books ? seg : kSpare];
  bool open = books;
  if constexpr (EXT) {
    bk.at = !books ? 0 : 2 * (last_e >= Q ? last_e - Q : last_e) + (last_e >= Q ? 1 : 0);
    bk.best = 4 * Book{}.clip_best;
    bk.i = bk.k = 0;
    bk.clip = S.flags & F_CLIP;
    bk.xd = 4 * min(max(S.xdrop, -(1 << 27)), 1 << 28);
    bk.pot4 = 4 * S.ext * (W - bl + (last_odd ? 1 : 0));
    bk.row4 = 8 * S.ext;
    bk.row0 = a1 - 4 - kw;         // the first row of the four steps before row step 0
    bk.m = m;
    bk.tail = n + bl - 2 * kw;     // rows after this: the band's last even cell lies past the text
    if constexpr (CUT) {
      bk.cut = 4 * Book{}.cut_best;
      bk.cut_row = cut + below;  // rows after this start past the cut
      bk.cut_tail = cut + bl - 2 * kw;
    }
  }
  // Row steps from which some cell lies past the text.
  const int32_t r_tail = __reduce_min_sync(FULL, has ? n + bl - kw - a1 : INT32_MAX);
  // Word k's cells: e and f are the gap values entering them; h their diagonal, then their H.
  auto cell = [&](int k, const uint32_t (&cb)[NC], uint32_t& h, uint32_t et, uint32_t ft,
                  uint32_t& eo, uint32_t& fo, uint32_t& ac) {
    const uint32_t c = cb[k >> 3] >> (4 * ((k & 7) >> 1));
    const uint32_t dg = (k & 1) ? (c & (4u * kW2)) * v1 + h : (c & kW2) * v4 + h;
    if constexpr (TB) {
      const uint32_t ec = et & 0xfffcfffcu, fc = and_or(ft, mlow, kone);
      const uint32_t ht = __vimax3_u16x2(dg, fc, ec);
      const uint32_t hs = and_or(ht, mlow, ktwo);
      const uint32_t y = pick(et, ft, msel);  // E opened << 1 | F extended
      ac = mad<16>(ac, y);
      ac = mad<-1>(ec, ac);
      ac = mad<4>(ht, ac);
      ac = mad<-4>(hs, ac);  // (winner - 2) << 2
      h = hs;
      eo = ec;
      fo = fc;
    } else {
      (void)ac;
      h = __vimax3_u16x2(dg, ft, et);
      eo = et;
      fo = ft;
    }
  };
  uint4* tbp = nullptr;
  if constexpr (TB) tbp = reinterpret_cast<uint4*>(a.tb + J.tb_word) + l;

  auto row_step = [&](int32_t r, auto tailtag) {
    constexpr bool TAIL = decltype(tailtag)::value;
    if ((r & 15) == 0) {
      if (r > 0) {
        T[NT] = __funnelshift_r(t0, t1, tsh);
        Pn = rev2(__funnelshift_r(p0, p1, psh));
      }
      // The chunk after this one.
      const int32_t xt = (tx + r + 16 * (NT + 1)) >> 4, xp = (px + 1 + r + 16) >> 4;
      t0 = word(J.t_word, xt, tlim);
      t1 = word(J.t_word, xt + 1, tlim);
      p0 = word(J.p_word, xp, plim);
      p1 = word(J.p_word, xp + 1, plim);
    }
    if (r <= rF) masks(r);
    // EXT, some columns past the text: cells e <= te lie in it (the odd step's: e < te).
    [[maybe_unused]] const int32_t te = n + bl - (a1 + r) - k0;
    auto in_text = [&](int k, int32_t t) -> uint32_t {
      return (k <= t ? 0xffffu : 0u) | (Q + k <= t ? 0xffff0000u : 0u);
    };
    [[maybe_unused]] uint32_t sM = 0, sK = 0, sC = 0;
    if constexpr (CUT) {
      sC = __shfl_up_sync(FULL, C[Q - 1], 1);
      if (leftmost) sC = kNegM;
    }
    if constexpr (EXT) {
      sM = __shfl_up_sync(FULL, M[Q - 1], 1);
      sK = __shfl_up_sync(FULL, MK[Q - 1], 1);
      if (leftmost) sM = kNegM;
    }
    uint32_t G[Q], cb[NC];
    // Even step: offsets 2k from their odd neighbours.
    matches(Me, cb);
#pragma unroll
    for (int k = 0; k < Q; ++k) G[k] = mad<1>(HB[k], mg2);
    {
      // What the last word's cells hand to the right: its low half to the lane's own word 0.
      const uint32_t er = __vmaxu2(G[Q - 1], E[Q - 1]);
      uint32_t el = __shfl_up_sync(FULL, er, 1);
      if (leftmost) el = kNegE;
      el = __byte_perm(el, er, 0x5432);
#pragma unroll
      for (int k = Q - 1; k >= 0; --k) {
        const uint32_t et = k ? __vmaxu2(G[k ? k - 1 : 0], E[k ? k - 1 : 0]) : el;
        const uint32_t ft = __vmaxu2(G[k], F[k]);
        cell(k, cb, HA[k], et, ft, E[k], F[k], acc[TB ? 2 * k : 0]);
      }
    }
#pragma unroll
    for (int q = 0; q < NT; ++q) T[q] = __funnelshift_r(T[q], T[q + 1], 2);
    T[NT] >>= 2;
    // Odd step: offsets 2k + 1 from their even neighbours.
    matches(Mo, cb);
#pragma unroll
    for (int k = 0; k < Q; ++k) G[k] = mad<1>(HA[k], mg2);
    {
      // What word 0's cells hand down to the left, likewise.
      const uint32_t fl = __vmaxu2(G[0], F[0]);
      uint32_t fr = __shfl_down_sync(FULL, fl, 1);
      if (rightmost) fr = kNegF;
      fr = __byte_perm(fl, fr, 0x5432);
#pragma unroll
      for (int k = 0; k < Q; ++k) {
        const uint32_t et = __vmaxu2(G[k], E[k]);
        const uint32_t ft =
            k + 1 < Q ? __vmaxu2(G[k + 1 < Q ? k + 1 : 0], F[k + 1 < Q ? k + 1 : 0]) : fr;
        cell(k, cb, HB[k], et, ft, E[k], F[k], acc[TB ? 2 * k + 1 : 0]);
      }
    }
    if constexpr (EXT) {
      uint32_t ml[Q], pl[Q];
      ml[0] = __byte_perm(sM, M[Q - 1], 0x5432);
      pl[0] = __byte_perm(sK, MK[Q - 1], 0x5432);
#pragma unroll
      for (int k = 1; k < Q; ++k) {
        ml[k] = M[k - 1];
        pl[k] = MK[k - 1];
      }
      if (any_even) {
        // An even last cell: what stands left of its pair, and the even cells.
        put_last(even_last[r & 3][0], ml);
        put_last(even_last[r & 3][1], pl);
        put_last(even_last[r & 3][2], HA);
      }
      if constexpr (CUT) {
        // Cells up to the cut (and the text's end): their largest, without its offset.
        const int32_t tc = min(n, cut) + bl - (a1 + r) - k0;
        uint32_t cl[Q];
        cl[0] = __byte_perm(sC, C[Q - 1], 0x5432);
#pragma unroll
        for (int k = 1; k < Q; ++k) cl[k] = C[k - 1];
        if (any_even) put_last(even_last[r & 3][3], cl);
#pragma unroll
        for (int k = Q - 1; k >= 0; --k) {
          uint32_t xa = mad<1>(HA[k], ha);
          if (k == 0) xa &= pad0;
          C[k] = mad<1>(__vimax3_u16x2(cl[k], xa & in_text(k, tc), HB[k] & in_text(k, tc - 1)), 2u * e4);
        }
        if (any_odd) put_last(odd_last[r & 3][3], C);
      }
#pragma unroll
      for (int k = Q - 1; k >= 0; --k) {
        uint32_t xa = mad<1>(HA[k], ha), xb = TB ? mad<1>(HB[k], hb) : HB[k];
        if (k == 0) xa &= pad0;
        if constexpr (TAIL) {
          xa &= in_text(k, te);
          xb &= in_text(k, te - 1);
        }
        row_max(xa, xb, mad<1>(kc0, (uint32_t)(2 * k) + ((uint32_t)(2 * (Q + k)) << 16)), ml[k], pl[k],
                M[k], MK[k]);
      }
      if (any_odd) {
        put_last(odd_last[r & 3][0], M);
        put_last(odd_last[r & 3][1], MK);
      }
    }
#pragma unroll
    for (int q = NT - 1; q > 0; --q) P[q] = __funnelshift_l(P[q - 1], P[q], 2);
    P[0] = __funnelshift_l(Pn, P[0], 2);
    Pn = mad<4>(Pn, 0u);
  };

  for (int32_t r = 0; r < Rtot;) {
    if (!EXT || r < r_tail)
      row_step(r, std::false_type{});
    else
      row_step(r, std::true_type{});
    ++r;
    if (EXT && (r & 3) == 0) {
      // The books of the four rows these steps finished (align.rs:2580-2640), in the lane that
      // holds the band's last cell; all lanes go along.
      const int32_t i0 = r + bk.row0, row4 = bk.row4, v0 = off - bk.pot4 - row4 * i0;
      const int32_t best = bk.best, xd = bk.xd;
      const bool clip = bk.clip;
      const uint16_t* const fs = reinterpret_cast<const uint16_t*>(last[0][0]) + bk.at;
      constexpr int kRow = 4 * kArray, kArray2 = 2 * kArray;
      constexpr uint32_t ha1 = TB ? ~0u : 1u;
      const uint32_t x4 = row4 / 2 + ha1;
      auto row_of = [&](int t, uint32_t& k) {
        uint32_t f = fs[t * kRow];
        k = fs[t * kRow + kArray] | (~f & 1u);
        if (any_even) {
          // An even last cell is yet to be counted, where it lies in the text.
          const uint32_t x = fs[t * kRow + kArray2] + x4;
          if (!last_odd && x > f && i0 + t <= bk.tail) {
            f = x;
            k = (uint32_t)(2 * kw);
          }
        }
        return (int32_t)f;
      };
      // A row's largest up to the cut.
      auto cut_of = [&](int t) {
        uint32_t f = fs[t * kRow + 3 * kArray];
        if (any_even && !last_odd && i0 + t <= min(bk.tail, bk.cut_tail))
          f = max(f, fs[t * kRow + kArray2] + x4);
        return (int32_t)(f & ~3u) + (v0 - t * row4);
      };
      // Together: the largest row, the first of equals (3 - t in the low bits), where no row can
      // end the pass.
      int32_t top = INT32_MIN, least = INT32_MAX;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        uint32_t f = fs[t * kRow];
        if (any_even) f = max(f, last_odd ? 0u : fs[t * kRow + kArray2] + x4);
        const int32_t v = (int32_t)and_or(f, ~3u, 3u - t) + (v0 - t * row4);
        top = max(top, v);
        least = min(least, v);
      }
      const bool slow = open && (i0 < 1 || i0 + 3 >= bk.m || i0 + 3 > bk.tail ||
                                 (clip && least - 3 + xd < max(best, top)));
      if (!__any_sync(FULL, slow)) {
        if (clip && (top & ~3) > best) {
          const int t = 3 - (top & 3);
          uint32_t pk;
          row_of(t, pk);
          bk.best = top & ~3;
          bk.i = i0 + t;
          bk.k = (int32_t)pk;
        }
        if constexpr (CUT) {
          int32_t c = bk.cut;
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (open && i0 + t <= bk.cut_row) c = max(c, cut_of(t));
          bk.cut = c;
        }
      } else {
#pragma unroll 1
        for (int t = 0; t < 4; ++t) {
          const int32_t i = i0 + t;
          uint32_t pk;
          const int32_t v = (row_of(t, pk) & ~3) + (v0 - t * row4);
          if (!open || i < 1) continue;
          const bool to_cut = CUT && i <= bk.cut_row;
          const int32_t vc = to_cut ? cut_of(t) : 0;
          if (to_cut && vc > bk.cut) bk.cut = vc;
          if (clip && v > bk.best) {
            bk.best = v;
            bk.i = i;
            bk.k = (int32_t)pk;
          }
          const bool stop = clip && v + xd < bk.best;
          if (stop || i == m) {
            const bool cell = clip && (S.flags & F_CELL) && bk.i;
            a.out[jid] = DRes{stop ? NEG : v >> 2, clip ? bk.best >> 2 : Book{}.clip_best,
                              CUT ? bk.cut >> 2 : 0, to_cut && !stop ? vc >> 2 : NEG,
                              stop ? 0u : (uint32_t)(i - bl) + pk, cell ? (uint32_t)bk.i : 0u,
                              cell ? (uint32_t)(bk.i - bl + bk.k) : 0u, (uint32_t)min(i + above, n),
                              (uint32_t)i, (uint32_t)i, band_cells(i, below, above, n)};
            open = false;
          }
        }
      }
    }
    if constexpr (TB) {
      if ((r & 3) == 0) {
        // Four row steps: one 16-byte store per quad of words, lane-fastest.
        if (has && own && r < N + 4) {
#pragma unroll
          for (int q = 0; q < Q / 2; ++q)
            tbp[q * L] = make_uint4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
          tbp += (Q / 2) * L;
        }
      }
    }
    if constexpr (EXT) {
      if (!TEAM && (r & 3) == 0 && !__any_sync(FULL, open)) break;
    }
    if (!EXT && r == next_end) {
      // Passes whose cell (m, n) this row step computed.
      const int32_t Kend = n - m + bl, ke = (Kend >> 1) - k0;
      if (has && own && r == N && ke >= 0 && ke < 2 * Q) {
        uint32_t u = 0;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const uint32_t h = (Kend & 1) ? HB[k] : HA[k];
          if (ke == k) u = h & 0xffffu;
          if (ke == Q + k) u = h >> 16;
        }
        DRes o{};
        o.score = (((int32_t)(u & ~3u) + off) >> 2) - S.ext * (m + n);
        o.cut_score = NEG;
        o.score_col = (uint32_t)n;
        o.text_read = (uint32_t)min(m + above, n);
        o.last_row = o.rows = (uint32_t)m;
        o.cells = band_cells(m, below, above, n);
        a.out[jid] = o;
      }
      next_end = __reduce_min_sync(FULL, has && N > r ? N : INT32_MAX);
    }
    if constexpr (TEAM) {
      if ((r & (2 * Q - 1)) == 0) {
        const int turn = (r / (2 * Q)) & 1;
        uint32_t v = 0;
        if ((r & (kWRebase - 1)) == 0) {
#pragma unroll
          for (int k = 0; k < Q; ++k) v = __vimax3_u16x2(v, HA[k], HB[k]);
          v = __reduce_max_sync(FULL, own ? max(v & 0xffffu, v >> 16) : 0u);
          if (lane == 0) X->top[turn][w] = v;
        }
        if ((lane == 30 && w < NW - 1) || (lane == 1 && w > 0)) {
          uint4* at = lane == 30 ? X->up[turn][w] : X->down[turn][w];
#pragma unroll
          for (int k = 0; k < Q; ++k) at[k] = make_uint4(HA[k], HB[k], E[k], F[k]);
          if constexpr (EXT)
            if (lane == 30)
#pragma unroll
              for (int k = 0; k < Q; ++k) X->row[turn][w][k] = make_uint2(M[k], MK[k]);
        }
        if (EXT && books) X->ended[turn] = !open;
        __syncthreads();
        if (EXT && X->ended[turn]) break;
        if ((lane == 0 && w > 0) || (lane == 31 && w < NW - 1)) {
          const uint4* at = lane == 0 ? X->up[turn][w - 1] : X->down[turn][w + 1];
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            const uint4 x = at[k];
            HA[k] = x.x;
            HB[k] = x.y;
            E[k] = x.z;
            F[k] = x.w;
          }
          if constexpr (EXT)
            if (lane == 0)
#pragma unroll
              for (int k = 0; k < Q; ++k) {
                const uint2 x = X->row[turn][w - 1][k];
                M[k] = x.x;
                MK[k] = x.y;
              }
        }
      }
    }
    if ((r & (kWRebase - 1)) == 0) {
      // Each pass's largest field back to the top.
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < Q; ++k) v = __vimax3_u16x2(v, HA[k], HB[k]);
      v = max(v & 0xffffu, v >> 16);
      if constexpr (TEAM) {
        const int turn = (r / (2 * Q)) & 1;
        v = X->top[turn][0];
        for (int u = 1; u < NW; ++u) v = max(v, X->top[turn][u]);
      } else {
        for (int s = 1; s < L; s <<= 1) {
          const uint32_t u = __shfl_down_sync(FULL, v, s);
          if (l + s < L) v = max(v, u);
        }
        v = __shfl_sync(FULL, v, min(seg * L, 31));
      }
      const int32_t delta = (int32_t)(v - kH) - wtop;
      const uint32_t dd = ((uint32_t)(-delta) & 0xffffu) * kW2;
#pragma unroll
      for (int k = 0; k < Q; ++k) {
        HA[k] = __viaddmax_u16x2(HA[k], dd, kNegH);
        HB[k] = __viaddmax_u16x2(HB[k], dd, kNegH);
        E[k] = __viaddmax_u16x2(E[k], dd, kNegE);
        F[k] = __viaddmax_u16x2(F[k], dd, kNegF);
        if constexpr (EXT) M[k] = __viaddmax_u16x2(M[k], dd, kNegM);
        if constexpr (CUT) C[k] = __viaddmax_u16x2(C[k], dd, kNegM);
      }
      off += delta;
    }
  }
  if constexpr (TB) {
    if constexpr (TEAM) {
      __syncthreads();
      if (w == 0) walk_wave<Q>(a, jid, true, L, 32, lane, 0, N);
    } else {
      __syncwarp();
      walk_wave<Q>(a, jid, has, L, L, l, min(seg * L, 31), N);
    }
  }
  __syncwarp();
}

template <int Q, bool TB, bool EXT, bool CUT>
__global__ void __launch_bounds__(128, sfk::wave_blocks(Q, TB, EXT)) wave16_kernel(sfk::AffLaunch a) {
  const int lane = threadIdx.x & 31;
  __shared__ WaveLast<Q, EXT> Z[4];
  // The first task by place; the queue hands out those after the grid's first ones.
  const uint32_t grid_tasks = (gridDim.x * blockDim.x) >> 5;
  // (Every q is a shuffle's: the compiler then keeps what follows from it in uniform registers.)
  uint32_t q = __shfl_sync(FULL, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, 0);
  while (q < a.njobs) {
    const uint2 task = a.tasks[q];
    const int L = (int)(task.y & 0xffu), np = (int)(task.y >> 8), seg = lane / L;
    const bool has = seg < np;
    wave_passes<Q, TB, EXT, false, CUT>(a, a.order[task.x + (has ? (uint32_t)seg : 0u)], has, L, lane, seg,
                                   Z[threadIdx.x >> 5], nullptr);
    if (a.njobs <= grid_tasks) break;
    uint32_t next = 0;
    if (lane == 0) next = atomicAdd(a.counter, 1u);
    q = __shfl_sync(FULL, grid_tasks + next, 0);
  }
}

// One pass per block of two to seven warps.
template <int Q, bool TB, bool EXT>
__global__ void __launch_bounds__(32 * sfk::wave_most_warps(Q), sfk::wave_team_blocks(Q, TB, EXT))
    wave16t_kernel(sfk::AffLaunch a) {
  __shared__ WaveTeam<Q, EXT> X;
  __shared__ WaveLast<Q, EXT> Z;
  uint32_t q = blockIdx.x;
  while (q < a.njobs) {
    const uint2 task = a.tasks[q];
    wave_passes<Q, TB, EXT, true, false>(a, a.order[task.x], true, (int)(task.y & 0xffu), threadIdx.x & 31,
                                    0, Z, &X);
    if (a.njobs <= gridDim.x) break;
    __syncthreads();
    if (threadIdx.x == 0) X.task = gridDim.x + atomicAdd(a.counter, 1u);
    __syncthreads();
    q = X.task;
  }
}

}  // namespace

namespace sfk {

template <int Q, bool EXT>
cudaError_t launch_wave16t_q(bool tb, const AffLaunch& a, int grid, int block, cudaStream_t s) {
  if (tb)
    wave16t_kernel<Q, true, EXT><<<grid, block, 0, s>>>(a);
  else
    wave16t_kernel<Q, false, EXT><<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

template <int Q>
cudaError_t launch_wave16c_q(const AffLaunch& a, int grid, cudaStream_t s) {
  wave16_kernel<Q, false, true, true><<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

template <int Q, bool EXT>
cudaError_t launch_wave16_q(bool tb, const AffLaunch& a, int grid, cudaStream_t s) {
  if (tb)
    wave16_kernel<Q, true, EXT, false><<<grid, 128, 0, s>>>(a);
  else
    wave16_kernel<Q, false, EXT, false><<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace sfk
