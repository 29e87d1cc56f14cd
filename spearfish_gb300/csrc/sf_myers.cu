// Myers' bit-parallel edit distance (align.rs:47-168): one pair per P lanes of a warp, or, for
// patterns of many blocks, per team of two or four warps (P = 64, 128).
//
// The pattern's 64-row blocks are spread over the pair's lanes, B consecutive blocks a lane.
// Within one text column the blocks form a chain (block b needs the horizontal delta leaving
// block b - 1), across columns each block depends only on itself, so the lanes run a diagonal
// pipeline: lane l is at column t - l at step t, and takes the delta that lane l - 1 left at
// step t - 1 with two shuffles.
//
//  - The pattern is aligned to the lanes' end: the free rows lie above it, as rows that change
//    nothing (Infix: rows that match every base, so the zeros of row 0 reach the pattern's first
//    row; Global and Prefix: rows that match none, through which row 0's +1 passes).  So every
//    block's last row is bit 63, a delta travels as the sign bits of the block's two delta
//    words, ready to shift into the next block, and the distance is read at one lane.
//  - Match masks sit in shared memory by code, a lane to its own banks: one 8-byte load a block
//    instead of the four logic instructions that derive them from bit planes.  A fifth code
//    matches only the free rows: with no delta entering, a column of it leaves a lane's state
//    as it is, so lanes wait for column 0 on it.
//  - A lane reads its own columns' bases (a 16-base word every 16 steps), so no base travels.
//  - A lane's deltas of 32 steps collect in two words; the distance and its least value over
//    the columns come from their bit counts once every 32 steps, a column a lane.
//
// A team's warps run 63 steps apart, so the 32 deltas that leave a warp in one chunk of 32 steps
// are exactly those its neighbour takes in the next: two words through shared memory and one
// block barrier a chunk.
//
// Bound: the ALU pipe: 22 instructions a block and step and about 12 a step besides.
//
// Every block of every column is computed (no Ukkonen band): the reference's cutoff is
// exact whenever the distance is <= k and reports None otherwise (align.rs:87-168, pinned by
// its tests `random_vs_naive` / `related_vs_naive`), so comparing the full-column distance
// with k gives the same Option<u32>.  The band's skipped blocks would save no time here: the
// lanes holding them still step every column their upper neighbours step.
//
// What does save time is the end of a capped Global or Prefix pair: once every cell of the
// lanes' current columns exceeds k + 1 (and row 0 does), every later cell exceeds k, since a
// path to it crosses those columns, or the one beside them where it steps down between two
// lanes; then the pair's answer is fixed: None (Global) or the best so far (Prefix).  Checked
// once every 32 steps from each lane's bottom score (the bit counts) less its +1 vertical
// deltas.  Between two warps of a team 32 columns lie open, so the bound is 32 higher there.
// Infix pairs never stop (row 0 is 0).
#include <type_traits>

#include "sf_internal.cuh"

namespace {

using sf::FULL;

constexpr int kCodes = 5;                    // A, C, G, T and "no column yet"
constexpr int kCodeBytes = 32 * 8;           // a code's masks: 8 bytes a lane
constexpr int kBlockBytes = kCodes * kCodeBytes;

// The low (hi) bits of the 16 codes of w, gathered into 16 bits.
__device__ __forceinline__ uint32_t gather16(uint32_t x) {
  x &= 0x55555555u;
  x = (x | (x >> 1)) & 0x33333333u;
  x = (x | (x >> 2)) & 0x0F0F0F0Fu;
  x = (x | (x >> 4)) & 0x00FF00FFu;
  return (x | (x >> 8)) & 0x0000FFFFu;
}

__device__ __forceinline__ int popc64(uint2 v) { return __popc(v.x) + __popc(v.y); }

// align.rs:50-66 `block` on 32-bit halves.  in_p / in_m: the words whose sign bits are the +1 /
// -1 delta entering the block; on return those of the delta leaving it.
__device__ __forceinline__ void myers_block(uint2& pv, uint2& mv, uint2 eq, uint32_t& in_p,
                                            uint32_t& in_m) {
  const uint32_t xvl = eq.x | mv.x, xvh = eq.y | mv.y;
  const uint32_t el = eq.x | (in_m >> 31);
  uint32_t sl, sh;
  asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, %5;"
      : "=&r"(sl), "=r"(sh)
      : "r"(el & pv.x), "r"(pv.x), "r"(eq.y & pv.y), "r"(pv.y));
  const uint32_t xl = (sl ^ pv.x) | el, xh = (sh ^ pv.y) | eq.y;
  const uint32_t pl = mv.x | ~(xl | pv.x), ph = mv.y | ~(xh | pv.y);
  const uint32_t ml = pv.x & xl, mh = pv.y & xh;
  const uint32_t spl = __funnelshift_l(in_p, pl, 1), sph = __funnelshift_l(pl, ph, 1);
  const uint32_t sml = __funnelshift_l(in_m, ml, 1), smh = __funnelshift_l(ml, mh, 1);
  pv.x = sml | ~(xvl | spl);
  pv.y = smh | ~(xvh | sph);
  mv.x = spl & xvl;
  mv.y = sph & xvh;
  in_p = ph;
  in_m = mh;
}

// Shared memory: the warps' match masks, then (teams) the chunk's words and votes by parity.
struct Team {
  uint32_t acc[2][4][2];
  uint32_t past[2][4];
  uint32_t task;
};

template <int B, bool TEAM>
__global__ void __launch_bounds__(128, B <= 2 ? 8 : (B == 3 ? 6 : 5)) myers_kernel(sfk::MyersLaunch a) {
  extern __shared__ uint64_t smem[];
  __shared__ Team X;
  const int lane = threadIdx.x & 31, w = TEAM ? threadIdx.x >> 5 : 0;
  const int W = TEAM ? blockDim.x >> 5 : 1;
  // A lane's masks: code c of block bb at byte bb * kBlockBytes + c * kCodeBytes + 8 * lane.
  const char* eqb = reinterpret_cast<const char*>(smem) +
                    (threadIdx.x >> 5) * (B * kBlockBytes) + lane * 8;
  char* eqw = const_cast<char*>(eqb);

  // The first task by place; the queue hands out those after the grid's first ones.
  const uint32_t grid_tasks = TEAM ? gridDim.x : (gridDim.x * blockDim.x) >> 5;
  uint32_t q = TEAM ? blockIdx.x : __shfl_sync(FULL, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, 0);
  for (bool more = q < a.ntasks; more;) {
    const uint2 task = a.tasks[q];
    const int P = TEAM ? 32 * W : (int)(task.y & 0xffu), np = TEAM ? 1 : (int)(task.y >> 8);
    const int seg = TEAM ? 0 : lane / P;
    const int l = TEAM ? 32 * w + lane : lane - seg * P;
    const bool has = seg < np;
    const uint32_t jid = a.order[task.x + (has ? (uint32_t)seg : 0u)];
    const sf::MJob J = a.jobs[jid];
    const int m = (int)J.m, n = (int)J.n;
    const bool infix = J.mode == 0, glob = J.mode == 2;
    const int free_rows = P * B * 64 - m;  // above the pattern

    uint2 pv[B], mv[B];
    const int plim = (m >> 4) + 1;
#pragma unroll
    for (int bb = 0; bb < B; ++bb) {
      const int row0 = (l * B + bb) * 64 - free_rows;  // the pattern row of bit 0
      uint32_t lo[2] = {0, 0}, hi[2] = {0, 0};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int x = row0 + 16 * h + 1;  // packed position (one leading pad base)
        const int i0 = min(max(x >> 4, 0), plim), i1 = min(max((x >> 4) + 1, 0), plim);
        const uint32_t u = __funnelshift_r(__ldg(a.pool + J.p_word + i0), __ldg(a.pool + J.p_word + i1),
                                           2 * (x & 15));
        lo[h >> 1] |= gather16(u) << (16 * (h & 1));
        hi[h >> 1] |= gather16(u >> 1) << (16 * (h & 1));
      }
      // Bits of free rows.
      const int f = min(max(-row0, 0), 64);
      const uint32_t fr[2] = {f >= 32 ? ~0u : (1u << f) - 1u,
                              f >= 64 ? ~0u : (f <= 32 ? 0u : (1u << (f - 32)) - 1u)};
#pragma unroll
      for (int c = 0; c < kCodes; ++c) {
        uint2 e;
        uint32_t* eh[2] = {&e.x, &e.y};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t k = (c & 1 ? lo[h] : ~lo[h]) & (c & 2 ? hi[h] : ~hi[h]);
          *eh[h] = c == 4 ? fr[h] : (k & ~fr[h]) | (infix ? fr[h] : 0u);
        }
        *reinterpret_cast<uint2*>(eqw + bb * kBlockBytes + c * kCodeBytes) = e;
      }
      pv[bb] = make_uint2(~fr[0], ~fr[1]);
      mv[bb] = make_uint2(0, 0);
    }
    __syncwarp();

    // Lane l is at column s - delay at step s.
    const int delay = TEAM ? 63 * w + lane : l;
    const int tlim = (n >> 4) + 1;
    auto bases = [&](int s) {  // the 16 columns from step s on
      const int x = s - delay + 1;
      const int i0 = min(max(x >> 4, 0), tlim), i1 = min(max((x >> 4) + 1, 0), tlim);
      return __funnelshift_r(__ldg(a.pool + J.t_word + i0), __ldg(a.pool + J.t_word + i1), 2 * (x & 15));
    };
    const int last = TEAM ? 63 * (W - 1) + 31 : P - 1;  // the delay of the pattern's last row
    const int mine = has && m > 0 && n > 0 ? (n - 1 + last) / 32 + 1 : 0;
    const int chunks = TEAM ? mine : (int)__reduce_max_sync(FULL, mine);

    int score = m, best = glob ? INT32_MAX : m;
    // This lane's bottom score in its current column (D[i][0] = i), for the cap.
    int bottom = max((l + 1) * B * 64 - free_rows, 0);
    const bool capped = a.kcut && has && !infix && (uint64_t)J.k < (uint64_t)m + (uint64_t)n;
    const int far = (int)min((uint64_t)J.k, (uint64_t)0x3fffffff) + (TEAM ? 34 : 2);
    const bool any_cap = __any_sync(FULL, capped);
    bool dead = false;
    uint32_t out_p = 0, out_m = 0;  // the deltas leaving this lane
    // What enters the pair's first lane: row 0's delta, or (teams) the last warp's words, a
    // column at their sign bit, moved on by a multiplication (the FMA pipe).
    const bool first = l == 0 || (TEAM && lane == 0);
    const bool relay = TEAM && w > 0;
    const uint32_t step_mul = relay ? 2u : 1u;
    uint32_t src_p = infix || relay ? 0u : 0x80000000u, src_m = 0;
    const uint32_t top = src_p;

    uint32_t tw = 0;  // the next 16 columns' bases
    auto chunk = [&](int s, auto filltag) {
      constexpr bool FILL = decltype(filltag)::value;
      uint32_t acc_p = 0, acc_m = 0;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        const uint32_t tn = bases(s + 16 * half + 16);
#pragma unroll(B <= 2 ? 4 : 2)
        for (int k = 0; k < 16; ++k) {
          uint32_t ip = __shfl_up_sync(FULL, out_p, 1), im = __shfl_up_sync(FULL, out_m, 1);
          uint32_t c = tw & 3u;
          if constexpr (FILL) {
            const bool wait = s + 16 * half + k < delay;
            if (wait) c = 4;
            if (first) {
              ip = wait && !relay ? 0u : src_p;
              im = src_m;
            }
          } else if (first) {
            ip = src_p;
            im = src_m;
          }
          if constexpr (TEAM) {
            src_p *= step_mul;
            src_m *= step_mul;
          }
          tw >>= 2;
          const char* at = eqb + c * kCodeBytes;
#pragma unroll
          for (int bb = 0; bb < B; ++bb)
            myers_block(pv[bb], mv[bb], *reinterpret_cast<const uint2*>(at + bb * kBlockBytes), ip, im);
          out_p = ip;
          out_m = im;
          acc_p = __funnelshift_l(ip, acc_p, 1);
          acc_m = __funnelshift_l(im, acc_m, 1);
        }
        tw = tn;
      }
      return make_uint2(acc_p, acc_m);
    };

    for (int ch = 0; ch < chunks; ++ch) {
      const int s = 32 * ch;
      uint2 acc = make_uint2(0, 0);
      if constexpr (TEAM) {
        // A warp whose first column is still to come leaves no deltas.
        if (s + 31 >= 63 * w) {
          if (s <= 63 * w) tw = bases(s);  // the warp's first chunk
          if (relay) {
            src_p = ch > 0 ? X.acc[(ch + 1) & 1][w - 1][0] : 0u;
            src_m = ch > 0 ? X.acc[(ch + 1) & 1][w - 1][1] : 0u;
          } else {
            src_p = top;
          }
          acc = s < 63 * w + 31 ? chunk(s, std::true_type{}) : chunk(s, std::false_type{});
        }
      } else {
        if (ch == 0) tw = bases(0);
        acc = ch == 0 ? chunk(s, std::true_type{}) : chunk(s, std::false_type{});
      }
      bottom += __popc(acc.x) - __popc(acc.y);
      // The pair's last lane holds the last row's deltas: columns s - last .. + 31, shared out
      // over the pair's lanes (all of the warp's, if it is the only pair).
      const int own = TEAM ? 31 : (np == 1 ? P - 1 : min(seg * P + P - 1, 31));
      const uint32_t op = __shfl_sync(FULL, acc.x, own), om = __shfl_sync(FULL, acc.y, own);
      if (!TEAM || w == W - 1) {
        const int c0 = s - last;
        for (int t = TEAM || np == 1 ? lane : l; t < 32; t += TEAM || np == 1 ? 32 : P) {
          const int c = c0 + t;
          if (c >= 0 && c < n && (!glob || c == n - 1))
            best = min(best, score + __popc(op >> (31 - t)) - __popc(om >> (31 - t)));
        }
        score += __popc(op) - __popc(om);
      }
      bool past = false;
      if (any_cap) {
        int ups = 0;
#pragma unroll
        for (int bb = 0; bb < B; ++bb) ups += popc64(pv[bb]);
        past = bottom - ups >= far && (!first || relay || s + 32 >= far);
      }
      if constexpr (TEAM) {
        if (lane == 31) {
          X.acc[ch & 1][w][0] = acc.x;
          X.acc[ch & 1][w][1] = acc.y;
        }
        const bool all = __all_sync(FULL, past);
        if (lane == 0) X.past[ch & 1][w] = all;
        __syncthreads();
        if (capped && ch + 1 < mine) {
          bool every = true;
          for (int u = 0; u < W; ++u) every = every && X.past[ch & 1][u];
          if (every) {
            dead = true;
            break;
          }
        }
      } else if (any_cap) {
        const uint32_t lanes = (P == 32 ? FULL : (1u << P) - 1u) << min(seg * P, 31);
        const uint32_t bal = __ballot_sync(FULL, past);
        if (capped && ch + 1 < mine && (bal & lanes) == lanes) dead = true;
        if (__all_sync(FULL, dead || ch + 1 >= mine)) break;
      }
    }
    if (dead && glob) best = INT32_MAX;
    if constexpr (TEAM) {
      best = __reduce_min_sync(FULL, best);
      if (w == W - 1 && lane == 0) {
        if (m == 0 || n == 0) best = m == 0 ? (glob ? n : 0) : m;
        a.out[jid] = (uint32_t)best <= J.k ? (uint32_t)best : 0xffffffffu;
      }
    } else {
      if (np == 1) {
        best = __reduce_min_sync(FULL, best);
      } else {
        for (int t = 1; t < P; t <<= 1) {
          const int o = __shfl_down_sync(FULL, best, t);
          if (l + t < P) best = min(best, o);
        }
      }
      if (has && l == 0) {
        if (m == 0 || n == 0) best = m == 0 ? (glob ? n : 0) : m;
        a.out[jid] = (uint32_t)best <= J.k ? (uint32_t)best : 0xffffffffu;
      }
      __syncwarp();
    }
    if (a.ntasks <= grid_tasks) break;
    if constexpr (TEAM) {
      if (threadIdx.x == 0) X.task = grid_tasks + atomicAdd(a.counter, 1u);
      __syncthreads();
      q = X.task;
      __syncthreads();
    } else {
      if (lane == 0) q = grid_tasks + atomicAdd(a.counter, 1u);
      q = __shfl_sync(FULL, q, 0);
    }
    more = q < a.ntasks;
  }
}

template <int B>
cudaError_t launch_b(const sfk::MyersLaunch& a, int grid, int block, cudaStream_t s) {
  const size_t sm = (size_t)(block / 32) * B * kBlockBytes;
  if (a.team)
    myers_kernel<B, true><<<grid, block, sm, s>>>(a);
  else
    myers_kernel<B, false><<<grid, block, sm, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

namespace sfk {

cudaError_t launch_myers(int b, const MyersLaunch& a, int grid, int block, cudaStream_t s) {
  switch (b) {
    case 1: return launch_b<1>(a, grid, block, s);
    case 2: return launch_b<2>(a, grid, block, s);
    case 3: return launch_b<3>(a, grid, block, s);
    case 4: return launch_b<4>(a, grid, block, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sfk
