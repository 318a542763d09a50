// Low-latency linear-gap DP for small batches: a block per pair.
//
// Move evaluation, downpass levels, Wagner steps and single pairs are batches
// of one to a few hundred pairs, where what counts is how long one pair takes.
// k_lin_dp4 (a warp per pair) is built for throughput: a lane's four rows lag
// the next lane's by 7 steps, strips of 128 rows follow one another at least
// 288 steps apart and the warp stages its own columns, about 95 cycles a
// step.  Here one warp sweeps the band by antidiagonals t = r + j and the
// eight other warps of the block prepare its costs:
//   * lane k owns the D diagonals i = D k .. D k + D - 1 of the band (i = j - r
//     - dlo), two cells to a register (16-bit halves, the values of
//     k_lin_dp4): E[q] holds i = 2q and 2q + D/2, O[q] the odd ones above
//     them.  An even step updates E from O, an odd one O from E: a cell's
//     align predecessor is its own diagonal's last value, insert the diagonal
//     below, delete the one above; only the lane's edge needs a shuffle and a
//     byte permute, so a step is one short dependency chain whatever D is (up to
//     D = 16 one exchange serves two steps, see team_step).
//   * the helpers look up the costs of the next 8 double steps, one (lane,
//     double step) each, and lay them out in shared memory as the main warp
//     reads them: the align costs of every register, and the one new insert
//     and delete word (the others move along the registers).
//   * cells outside the band are forced to infinity by the mask that clears
//     the rank bits; cells outside the matrix have a pad character of cost 0
//     on one side, so infinity stays infinity and no edge needs a test.
// Values, ranks (the move backtrack_2d takes among tied ones) and the 16-bit
// condition are k_lin_dp4's, see linear4.cu; the band and results the
// reference's (algn.c:375-968, 3551-3666).
//
// Bound: the latency of a double step (shuffle, then permute, add-min and clear
// twice: 55 cycles, 82 measured with 8 diagonals a lane and 107 with 16), L1 + L2
// halves of them.  An exchange and late costs at each step took 93 and 126: one
// alignment of 1,500 bp 174 us, now 146.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include "poyd_internal.h"
#include "linear_kernels.cuh"

namespace poyd {
namespace {

constexpr unsigned kTFull = 0xffffffffu;
constexpr uint32_t kTInf2 = 0xC000C000u;
// Warp 0 sweeps; the warps w with w % 4 != 0 below 11 are its eight helpers: a
// scheduler of their own each, so that warp 0 issues alone (warps 4 and 8
// only write results).
constexpr int kTThreads = 32 * 11;
constexpr int kTChunk = 8;                      // double steps per chunk
constexpr int kTStride = 36;                    // bytes per row of the cost table
constexpr int kTPadChar = 32;
constexpr int kTWalk = 64;                      // chunks in the walk's window

template <int D>
struct TeamDim {
  static constexpr int NQ = D / 4;              // registers per parity
  static constexpr int NV = D / 8;              // 16-byte cost vectors per double step and lane
  static constexpr int kPad = 16 * D + 16;      // characters before and after a sequence
  static constexpr uint32_t kStep = NV * 512 + 256 + 64;  // bytes per double step (64: banks)
  static constexpr uint32_t kSlot = kTChunk * kStep;
  static constexpr uint32_t kRing = 2 * kSlot;
  static constexpr uint32_t kTab = kRing;                        // cost table
  static constexpr uint32_t kG = kTab + 33 * kTStride + 12;      // insert, delete costs [2][36] u16
  static constexpr uint32_t kMed = kG + 2 * 36 * 2;
  static constexpr uint32_t kEnd = kMed + 1024;                  // final registers [NQ][32]
  static constexpr uint32_t kSeq = kEnd + NQ * 128;              // the two sequences, padded
  // then the path, a byte per column (at most the slot's capacity)
  __host__ __device__ static constexpr uint32_t path(int sum) { return kSeq + (uint32_t)sum + 4 * kPad; }
  static constexpr uint32_t bytes(int mode, int sum) {
    return path(sum) + (mode == kDpChoice ? (uint32_t)sum + 16 : 16);
  }
  static_assert(kTWalk * 3 * (D / 2) * 4 <= (int)kRing, "the walk's window fits the ring");
};

struct TeamArgs {
  int n;
  const uint8_t *seq;
  const LinPlan *plans;
  const DevTables *tables;
  int gap;
  uint32_t *dm;
  int64_t dm_stride;  // words per pair
  int32_t *cost;
  LinTbArgs tb;
  DpK k;
};

__device__ __forceinline__ uint32_t t_prmt(uint32_t a, uint32_t b, uint32_t s) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}
__device__ __forceinline__ uint32_t t_mad(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Where a pair's cells are: dlo lowered to an even diagonal below the band, the
// band's indices [lo, hi), lo 1 or 2.  Index 0 and the last (hi <= 32 D - 1) are
// masked, so that the lanes' ring shuffles bring the first and the last lane
// an infinite neighbour.
struct TeamGeo {
  int L1, L2, dlo, lo, hi;
  int r0, j0;  // row and column of lane 0's first cell at double step 0
  int me;      // double step of the final cell
};
__device__ __forceinline__ TeamGeo team_geo(const LinPlan &P) {
  TeamGeo g;
  g.L1 = P.l1, g.L2 = P.l2;
  g.lo = 2 - (P.dlo & 1);
  g.dlo = P.dlo - g.lo;
  g.hi = P.wd + g.lo;
  g.r0 = -(g.dlo >> 1);
  g.j0 = g.dlo >> 1;
  g.me = (P.l1 + P.l2 - 2) >> 1;
  return g;
}

template <int MODE, int D>
struct TeamState {
  static constexpr int NQ = D / 4;
  uint32_t E[NQ], O[NQ], gi[NQ], gd[NQ];
  uint32_t kE[NQ], iE[NQ], kO[NQ], iO[NQ];  // masks: bits kept, infinity forced
  uint32_t aE[NQ], aO[NQ];                  // the moves of 8 steps
  uint32_t hE, kH, iH;  // high half: the next lane's first cell, its masks
};

// Appends a register's moves (the two low bits of x's halves; y is x with them
// cleared and the cells outside the band forced) to acc: as x - y, on the
// multiply-add pipe, where a forced low half never shares the register with a
// cell of the band (its borrow would reach the high half), i.e. but for q = 0.
__device__ __forceinline__ uint32_t team_move(uint32_t acc, uint32_t x, uint32_t y, int q,
                                              const DpK &K) {
  if (q == 0) return t_mad(acc, (uint32_t)K.four, x & 0x00030003u);
  return t_mad(y, (uint32_t)K.m1, t_mad(acc, (uint32_t)K.four, x));
}

// A lane's costs of one double step, as the helpers left them.
template <int D>
struct TeamCost {
  uint32_t W[D / 2], hW;
  uint2 g;
};
template <int D>
__device__ __forceinline__ void team_load(TeamCost<D> &C, const uint8_t *step, int lane) {
  const uint4 *cv = reinterpret_cast<const uint4 *>(step) + lane;
#pragma unroll
  for (int v = 0; v < D / 8; ++v) {
    const uint4 x = cv[32 * v];
    C.W[4 * v] = x.x, C.W[4 * v + 1] = x.y, C.W[4 * v + 2] = x.z, C.W[4 * v + 3] = x.w;
  }
  C.hW = reinterpret_cast<const uint32_t *>(cv)[4];  // the next lane's; lane 31: any (masked)
  C.g = reinterpret_cast<const uint2 *>(step + D / 8 * 512)[lane];
}

// One double step.  A lane also computes the next lane's first even cell, which
// its last odd one reads, so that all it needs of others is their odd cells of
// the double step before: one shuffle latency for two steps (not with 32
// diagonals a lane, which fill the two by themselves: the costs of a pair of
// 4,000 bp take 347 us, 384 with the extra cell).  cap: the final cell is in this
// one (0 even, 1 odd step): its registers go to `end`.
template <int MODE, int D>
__device__ __forceinline__ void team_step(TeamState<MODE, D> &S, const TeamCost<D> &C, int lane,
                                          const DpK &K, int cap, uint32_t *end) {
  constexpr int NQ = D / 4;
  const uint32_t(&W)[2 * NQ] = C.W;
  const uint2 g = C.g;
  const uint32_t hW = C.hW;
  const uint32_t below = __shfl_sync(kTFull, S.O[NQ - 1], lane + 31);  // lane - 1, in a ring
  constexpr bool kHalo = D < 32;
  const uint32_t above = kHalo ? __shfl_sync(kTFull, S.O[0], lane + 1) : 0u;
  const uint32_t one = (uint32_t)K.one;
  const uint32_t hd = S.gd[NQ - 1];
#pragma unroll
  for (int q = NQ - 1; q > 0; --q) S.gd[q] = S.gd[q - 1];
  S.gd[0] = g.y;
  uint32_t rw;
  {
    // the next lane's first cell, in the high half (the low one holds anything)
    uint32_t h = t_mad(hW, (uint32_t)K.k64, S.hE);
    h = __viaddmin_u16x2(S.O[NQ - 1], g.x, h);
    h = __viaddmin_u16x2(t_mad(above, (uint32_t)K.k64, 0), hd, h);
    h = (h & S.kH) | S.iH;
    const uint32_t lw = t_prmt(below, S.O[NQ - 1], 0x5432);
#pragma unroll
    for (int e = 0; e < NQ; ++e) {
      const int q = kHalo ? NQ - 1 - e : e;  // what waits for a shuffle last, or goes into one first
      uint32_t x = kHalo ? __viaddmin_u16x2(S.O[q], S.gd[q], t_mad(S.E[q], one, W[q]))
                         : __viaddmin_u16x2(S.E[q], W[q], t_mad(S.O[q], one, S.gd[q]));
      x = __viaddmin_u16x2(q ? S.O[q - 1] : lw, S.gi[q], x);
      S.E[q] = (x & S.kE[q]) | S.iE[q];
      if (MODE == kDpChoice) S.aE[q] = team_move(S.aE[q], x, S.E[q], q, K);
    }
    const uint32_t next = __shfl_sync(kTFull, S.E[0], lane + 1);
    if (kHalo) S.hE = t_mad(next, (uint32_t)K.k64, 0);
    rw = kHalo ? t_prmt(S.E[0], h, 0x7632) : t_prmt(S.E[0], next, 0x5432);
  }
  if (cap == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) end[32 * q + lane] = S.E[q];
  }
#pragma unroll
  for (int q = 0; q + 1 < NQ; ++q) S.gi[q] = S.gi[q + 1];
  S.gi[NQ - 1] = g.x;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    uint32_t x = kHalo ? __viaddmin_u16x2(S.E[q], S.gi[q], t_mad(S.O[q], one, W[NQ + q]))
                       : __viaddmin_u16x2(S.O[q], W[NQ + q], t_mad(S.E[q], one, S.gi[q]));
    x = __viaddmin_u16x2(q + 1 < NQ ? S.E[q + 1] : rw, S.gd[q], x);
    S.O[q] = (x & S.kO[q]) | S.iO[q];
    if (MODE == kDpChoice) S.aO[q] = team_move(S.aO[q], x, S.O[q], q, K);
  }
  if (cap == 1) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) end[32 * q + lane] = S.O[q];
  }
}

// The path of one pair by one warp: tb_pair4_solo's walk (linear4.cu) over this
// layout's moves, one byte per column (0 both characters, 1 the column's only,
// 2 the row's only) into `path`, last column first.  A diagonal run stays on
// one lane's words, so the window holds kTWalk chunks of that lane and its two
// neighbours.  Returns the number of columns, -1 when the path left the band.
template <int D>
__device__ __forceinline__ int team_walk(const LinPlan &P, bool swaped, int64_t cap,
                                         const uint32_t *dm, uint4 *win, uint8_t *path, int lane) {
  constexpr int NQ = D / 4, NV = D / 8;
  const TeamGeo g = team_geo(P);
  const uint4 *dm4 = reinterpret_cast<const uint4 *>(dm);
  const uint32_t *win4 = reinterpret_cast<const uint32_t *>(win);
  const int nch = g.me / kTChunk + 1;
  int r = P.l1 - 1, j = P.l2 - 1;
  int n = 0, wlo = nch, wk = 0;  // window: chunks [wlo, wlo + kTWalk), lanes [wk, wk + 3)
  while (r > 0 || (r == 0 && j >= 0)) {
    const int i = j - r - g.dlo;
    if (j < 0 || i < g.lo || i >= g.hi || n + 2 >= cap) return -1;  // left the band: a bug
    const int k = i / D, c = (i % D) >> 1, par = i & 1;
    const int w = par * NQ + c % NQ, sh0 = 16 * (c / NQ);
    const int m0 = (r + j) >> 1;
    if (m0 / kTChunk < wlo || k < wk || k >= wk + 3) {
      wlo = max(m0 / kTChunk - kTWalk + 1, 0);
      wk = max(k - 1, 0);
      __syncwarp();
      for (int e = lane; e < kTWalk * NV * 3; e += 32) {  // [chunk][vector][lane]
        const int ch = wlo + e / (3 * NV), v = e / 3 % NV, kk = wk + e % 3;
        if (ch < nch && kk < 32) win[e] = __ldcg(dm4 + ((int64_t)ch * NV + v) * 32 + kk);
      }
      __syncwarp();
    }
    // lane l: the move of cell (r - l, j - l); 4 = not read
    const int m = m0 - lane;
    uint32_t code = 4;
    if (r >= lane && j >= lane && n + lane + 2 < cap && m / kTChunk >= wlo) {
      const uint32_t x = win4[(((m / kTChunk - wlo) * NV + (w >> 2)) * 3 + (k - wk)) * 4 + (w & 3)];
      code = (x >> (2 * (7 - m % kTChunk) + sh0)) & 3u;
    }
    const uint32_t stop = __ballot_sync(kTFull, code != 0);
    const int f = stop ? __ffs(stop) - 1 : 32;  // lanes below f move diagonally
    const uint32_t cf = __shfl_sync(kTFull, code, f & 31);
    const int step = f < 32 && cf != 4;         // lane f's cell was read: its move too
    const int move_f = step ? (((cf == 1u) == swaped) ? 1 : 2) : 0;
    if (lane < f + step) path[n + lane] = (uint8_t)(lane == f ? move_f : 0);
    n += f + step;
    r -= f + (step && move_f != 1);
    j -= f + (step && move_f != 2);
  }
  return n;
}

// The outputs of the path by the whole block (ancestor_2, median_2_with_gaps):
// a thread takes consecutive columns; two block scans place its rows and
// columns of the sequences and its part of the gap-free median.
__device__ __forceinline__ void team_write(const LinTbArgs &A, const uint8_t *med, int id,
                                           const LinPlan &P, const uint8_t *s1, const uint8_t *s2,
                                           const uint8_t *path, int n, int64_t *scan) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int la = P.swap ? P.l2 : P.l1, lb = P.swap ? P.l1 : P.l2;
  const int64_t cap = slot_cap(la, lb);
  uint8_t *oa = A.out + A.out_off[id];
  uint8_t *ob = oa + cap, *ow = ob + cap, *om = ow + cap;
  if (n < 0) {
    if (tid == 0) A.out_len[2 * id] = A.out_len[2 * id + 1] = -1;
    return;
  }
  // inclusive sum over the block's threads
  auto block_scan = [&](int64_t v, int64_t *total) {
    int64_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(kTFull, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) scan[warp] = x;
    __syncthreads();
    int64_t before = 0, all = 0;
    for (int w = 0; w < kTThreads / 32; ++w) {
      before += w < warp ? scan[w] : 0;
      all += scan[w];
    }
    *total = all;
    return before + x;
  };
  const int per = (n + kTThreads - 1) / kTThreads, c0 = min(n, tid * per), c1 = min(n, c0 + per);
  int64_t both = 0, total;
  for (int c = c0; c < c1; ++c) both += (int64_t)(path[c] != 1) << 32 | (path[c] != 2);
  const int64_t before = block_scan(both, &total) - both;
  const int r0 = P.l1 - 1 - (int)(before >> 32), j0 = P.l2 - 1 - (int)(before & 0xffffffff);
  int kept = 0;
  for (int c = c0, r = r0, j = j0; c < c1; ++c) {
    const int mv = path[c];
    const int cr = mv != 1 ? (int)s1[r] : A.gap, cc = mv != 2 ? (int)s2[j] : A.gap;
    r -= mv != 1;
    j -= mv != 2;
    const int ca = P.swap ? cc : cr, cb = P.swap ? cr : cc, md = med[(ca << 5) | cb];
    oa[cap - 1 - c] = (uint8_t)ca;
    ob[cap - 1 - c] = (uint8_t)cb;
    ow[cap - 1 - c] = (uint8_t)md;
    kept += md != A.gap;
  }
  int64_t nm;
  int at = (int)(block_scan(kept, &nm) - kept);
  for (int c = c0, r = r0, j = j0; c < c1; ++c) {
    const int mv = path[c];
    const int cr = mv != 1 ? (int)s1[r] : A.gap, cc = mv != 2 ? (int)s2[j] : A.gap;
    r -= mv != 1;
    j -= mv != 2;
    const int md = med[P.swap ? (cc << 5) | cr : (cr << 5) | cc];
    if (md != A.gap) om[cap - 1 - at++] = (uint8_t)md;
  }
  if (tid == 0) {
    om[cap - 1 - nm] = (uint8_t)A.gap;  // ancestor_2 ends with the leading gap (algn.c:4140-4141)
    A.out_len[2 * id] = n;
    A.out_len[2 * id + 1] = (int32_t)nm + 1;
  }
}

template <int MODE, int D>
__global__ void __launch_bounds__(kTThreads) k_lin_team(const __grid_constant__ TeamArgs A) {
  using Dm = TeamDim<D>;
  constexpr int NQ = Dm::NQ, NV = Dm::NV;
  constexpr int sc = MODE == kDpChoice ? 4 : 1;
  extern __shared__ __align__(16) uint8_t team_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int id = blockIdx.x;
  const LinPlan P = A.plans[id];
  uint8_t *tab = team_sm + Dm::kTab, *med = team_sm + Dm::kMed;
  uint16_t *gi_t = reinterpret_cast<uint16_t *>(team_sm + Dm::kG), *gd_t = gi_t + 36;
  if (P.empty) {  // DOS.median: the non-empty (or second) sequence is the median
    if (MODE == kDpChoice) {
      const int la = P.swap ? P.l2 : P.l1, lb = P.swap ? P.l1 : P.l2;
      const int64_t cap = slot_cap(la, lb);
      const bool a_empty = P.empty == 1;
      const uint8_t *src = A.seq + ((a_empty != (bool)P.swap) ? P.s2_off : P.s1_off);
      const int len = a_empty ? lb : la;
      uint8_t *om = A.tb.out + A.tb.out_off[id] + 4 * cap - len;
      for (int i = tid; i < len; i += kTThreads) om[i] = src[i];
      if (tid == 0) {
        A.tb.out_len[2 * id] = 0;
        A.tb.out_len[2 * id + 1] = len;
      }
    }
    if (tid == 0) A.cost[id] = 0;
    return;
  }
  const TeamGeo g = team_geo(P);
  const bool swaped = !P.swap;  // backtrack priority (algn.c:3605-3666)
  const int rank_i = MODE == kDpChoice ? (swaped ? 1 : 2) : 0;
  const int rank_d = MODE == kDpChoice ? 3 - rank_i : 0;
#pragma unroll
  for (int e0 = 0; e0 < 33 * 33; e0 += kTThreads) {
    const int e = e0 + tid;
    if (e >= 33 * 33) break;
    const int a = e / 33, b = e - 33 * a;
    tab[a * kTStride + b] =
        a < 32 && b < 32 ? (uint8_t)(sc * (A.tables->packed[(a << 5) | b] & 0xffffu)) : 0;
  }
  if (tid < 33) {
    gi_t[tid] = (uint16_t)((tid < 32 ? sc * (A.tables->packed[tid] >> 16) : 0) + rank_i);
    gd_t[tid] = (uint16_t)((tid < 32 ? sc * (A.tables->packed[(tid << 5) | A.gap] & 0xffffu) : 0) + rank_d);
  }
  if (MODE == kDpChoice)
    for (int i = tid; i < 256; i += kTThreads)
      reinterpret_cast<uint32_t *>(med)[i] = reinterpret_cast<const uint32_t *>(A.tables->median)[i];
  uint8_t *s1 = team_sm + Dm::kSeq + Dm::kPad, *s2 = s1 + g.L1 + 2 * Dm::kPad;
#pragma unroll 4
  for (int x = tid; x < g.L1 + 2 * Dm::kPad; x += kTThreads) {
    const int r = x - Dm::kPad;
    s1[r] = r >= 0 && r < g.L1 ? A.seq[P.s1_off + r] : (uint8_t)kTPadChar;
  }
#pragma unroll 4
  for (int x = tid; x < g.L2 + 2 * Dm::kPad; x += kTThreads) {
    const int j = x - Dm::kPad;
    s2[j] = j >= 0 && j < g.L2 ? A.seq[P.s2_off + j] : (uint8_t)kTPadChar;
  }
  __syncthreads();

  // a helper's share of chunk c: lane k, double step 8 c + (lane >> 2)
  auto produce = [&](int c) {
    const int k = 4 * (warp - 1 - warp / 4) + (lane & 3), v = lane >> 2, m = kTChunk * c + v;
    const int r0 = g.r0 + m - 2 * NQ * k, j0 = g.j0 + m + 2 * NQ * k;
    const uint8_t *pa = s1 + r0, *pb = s2 + j0;
    int b[2 * NQ + 1];
#pragma unroll
    for (int x = 0; x <= 2 * NQ; ++x) b[x] = pb[x];
    uint32_t w[2 * NQ];
    uint32_t dlo = 0, dhi = 0;
#pragma unroll
    for (int x = 0; x < 2 * NQ; ++x) {
      const int ca = pa[-x];
      if (x == 0) dlo = gd_t[ca];
      if (x == NQ) dhi = gd_t[ca];
      const uint8_t *row = tab + ca * kTStride;
      const uint32_t ce = row[b[x]], co = row[b[x + 1]];
      if (x < NQ) {
        w[x] = ce;
        w[NQ + x] = co;
      } else {
        w[x - NQ] |= ce << 16;
        w[x] |= co << 16;
      }
    }
    uint8_t *o = team_sm + (c & 1) * Dm::kSlot + v * Dm::kStep;
    uint4 *cv = reinterpret_cast<uint4 *>(o) + k;
#pragma unroll
    for (int x = 0; x < NV; ++x) cv[32 * x] = make_uint4(w[4 * x], w[4 * x + 1], w[4 * x + 2], w[4 * x + 3]);
    reinterpret_cast<uint2 *>(o + NV * 512)[k] =
        make_uint2((uint32_t)gi_t[b[NQ]] | (uint32_t)gi_t[b[2 * NQ]] << 16, dlo | dhi << 16);
  };

  const int nch = g.me / kTChunk + 1;
  const int fcell = g.L2 - g.L1 - g.dlo, fk = fcell / D;  // the final cell's index and lane
  TeamState<MODE, D> S;
  uint4 *dm4 = MODE == kDpChoice ? reinterpret_cast<uint4 *>(A.dm + id * A.dm_stride) + lane : nullptr;
  uint32_t *end = reinterpret_cast<uint32_t *>(team_sm + Dm::kEnd);
  if (warp == 0) {
    const int r0 = g.r0 - 2 * NQ * lane, j0 = g.j0 + 2 * NQ * lane;
    const uint32_t keep = MODE == kDpChoice ? 0xFFFCu : 0xFFFFu;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      S.gi[q] = (uint32_t)gi_t[s2[j0 + q]] | (uint32_t)gi_t[s2[j0 + q + NQ]] << 16;
      S.gd[q] = (uint32_t)gd_t[s1[r0 - 1 - q]] | (uint32_t)gd_t[s1[r0 - 1 - q - NQ]] << 16;
      S.kE[q] = S.iE[q] = S.kO[q] = S.iO[q] = 0;
      S.E[q] = S.O[q] = kTInf2;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = D * lane + 2 * (q + h * NQ);
        const bool e = i >= g.lo && i < g.hi, o = i + 1 >= g.lo && i + 1 < g.hi;
        S.kE[q] |= (e ? keep : 0u) << (16 * h);
        S.iE[q] |= (e ? 0u : 0xC000u) << (16 * h);
        S.kO[q] |= (o ? keep : 0u) << (16 * h);
        S.iO[q] |= (o ? 0u : 0xC000u) << (16 * h);
        // the seed: cell (-1, -1), the align predecessor of (0, 0), is 0
        if (i == -g.dlo) S.E[q] &= h ? 0x0000FFFFu : 0xFFFF0000u;
      }
      S.aE[q] = S.aO[q] = 0;
    }
    const int ih = D * lane + D;
    const bool eh = ih >= g.lo && ih < g.hi;
    S.kH = eh ? keep << 16 : 0u;
    S.iH = eh ? 0u : 0xC0000000u;
    S.hE = __shfl_sync(kTFull, S.E[0], lane + 1) << 16;
  } else if (warp % 4) {
    produce(0);
  }
  __syncthreads();
  for (int c = 0; c < nch; ++c) {
    if (warp % 4) {
      if (c + 1 < nch) produce(c + 1);
    } else if (warp == 0) {
      const uint8_t *slot = team_sm + (c & 1) * Dm::kSlot;
      if (c + 1 < nch) {
        constexpr int kAhead = D < 32 ? 1 : 0;  // double steps a cost is read ahead
        TeamCost<D> C[2];
        if (kAhead) team_load<D>(C[0], slot, lane);
#pragma unroll
        for (int v = 0; v < kTChunk; ++v) {
          const int x = v + kAhead;
          if (x < kTChunk) team_load<D>(C[x & 1], slot + x * Dm::kStep, lane);
          team_step<MODE, D>(S, C[v & 1], lane, A.k, -1, end);
        }
      } else {
#pragma unroll 1
        for (int v = 0; v < kTChunk; ++v) {
          TeamCost<D> C;
          team_load<D>(C, slot + v * Dm::kStep, lane);
          team_step<MODE, D>(S, C, lane, A.k, v == g.me % kTChunk ? (fcell & 1) : -1, end);
        }
      }
      if (MODE == kDpChoice) {
        uint32_t w[2 * NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) w[q] = S.aE[q], w[NQ + q] = S.aO[q], S.aE[q] = S.aO[q] = 0;
#pragma unroll
        for (int x = 0; x < NV; ++x)
          dm4[((int64_t)c * NV + x) * 32] = make_uint4(w[4 * x], w[4 * x + 1], w[4 * x + 2], w[4 * x + 3]);
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    const int cc = (fcell % D) >> 1;
    const uint32_t v = (end[32 * (cc % NQ) + fk] >> (16 * (cc / NQ))) & 0xFFFFu;
    A.cost[id] = ((int)v - (int)tab[s1[0] * kTStride + s2[0]]) / sc;
  }
  if (MODE == kDpChoice) {
    __shared__ int s_n;
    __shared__ int64_t scan[kTThreads / 32];
    uint8_t *path = team_sm + Dm::path(g.L1 + g.L2);
    if (warp == 0) {
      const int n = team_walk<D>(P, swaped, slot_cap(g.L1, g.L2), A.dm + id * A.dm_stride,
                                 reinterpret_cast<uint4 *>(team_sm), path, lane);
      if (lane == 0) s_n = n;
    }
    __syncthreads();
    team_write(A.tb, med, id, P, s1, s2, path, s_n, scan);
  }
}

template <int MODE, int D>
int team_launch(const TeamArgs &A, int maxsum, cudaStream_t st) {
  static std::atomic<uint32_t> opted[64];
  const uint32_t sm = TeamDim<D>::bytes(MODE, maxsum);
  int dev = 0;
  cudaGetDevice(&dev);
  if (opted[dev & 63].load() < sm) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_lin_team<MODE, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTeamSmemMax);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_lin_team)");
    opted[dev & 63].store(kTeamSmemMax);
  }
  k_lin_team<MODE, D><<<A.n, kTThreads, sm, st>>>(A);
  return POYD_OK;
}

}  // namespace

// Diagonals per lane for bands up to maxwd (three more: the masked ends and the
// parity), 0 when the band or the sequences do not fit.
int lin_team_width(int maxwd, int maxsum) {
  const int d = maxwd + 3 <= 256 ? 8 : maxwd + 3 <= 512 ? 16 : maxwd + 3 <= 1024 ? 32 : 0;
  const uint32_t sm = d == 8 ? TeamDim<8>::bytes(kDpChoice, maxsum)
                    : d == 16 ? TeamDim<16>::bytes(kDpChoice, maxsum)
                    : d == 32 ? TeamDim<32>::bytes(kDpChoice, maxsum) : 0;
  return sm <= kTeamSmemMax ? d : 0;
}

int64_t lin_team_words(int width, int maxsum) {
  // (l1 + l2 - 2) / 2 + 1 double steps, whole chunks of width / 2 words a lane
  return ((int64_t)(maxsum / 2) / kTChunk + 1) * 32 * (width / 2);
}

int launch_lin_team(const LinDpArgs &D, int mode, int width, int64_t dm_stride, int maxsum,
                    cudaStream_t st) {
  TeamArgs A;
  A.n = D.n; A.seq = D.seq; A.plans = D.plans; A.tables = D.tables; A.gap = D.gap;
  A.dm = D.dm; A.dm_stride = dm_stride; A.cost = D.cost; A.tb = D.tb; A.k = D.k;
  if (mode == kDpChoice)
    return width == 8 ? team_launch<kDpChoice, 8>(A, maxsum, st)
         : width == 16 ? team_launch<kDpChoice, 16>(A, maxsum, st)
                       : team_launch<kDpChoice, 32>(A, maxsum, st);
  return width == 8 ? team_launch<kDpCost, 8>(A, maxsum, st)
       : width == 16 ? team_launch<kDpCost, 16>(A, maxsum, st)
                     : team_launch<kDpCost, 32>(A, maxsum, st);
}

}  // namespace poyd
