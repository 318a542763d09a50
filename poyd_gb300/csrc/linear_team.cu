// Low-latency linear-gap DP for small batches: a block per pair.
//
// Move evaluation, downpass levels, Wagner steps and single pairs are batches
// of one to a few hundred pairs, where what counts is how long one pair takes.
// k_lin_dp4 (a warp per pair) is built for throughput: a lane's four rows lag
// the next lane's by 7 steps, strips of 128 rows follow one another at least
// 288 steps apart and the warp stages its own columns, about 95 cycles a
// step.  Here one warp sweeps the band by antidiagonals t = r + j and the
// other eight warps of the block prepare its costs:
//   * lane k owns the D diagonals i = D k .. D k + D - 1 of the band (i = j - r
//     - dlo), two cells to a register (16-bit halves, the values of
//     k_lin_dp4): E[q] holds i = 2q and 2q + D/2, O[q] the odd ones above
//     them.  An even step updates E from O, an odd one O from E: a cell's
//     align predecessor is its own diagonal's last value, insert the diagonal
//     below, delete the one above; only the lane's edge needs a shuffle and a
//     byte permute, so a step is one short dependency chain whatever D is.
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
// Bound: the latency of a step (shuffle, permute, add-min, clear), L1 + L2 of
// them.
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
constexpr int kTHelpers = 8;                    // helper warps
constexpr int kTThreads = 32 * (1 + kTHelpers);
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
  static constexpr uint32_t bytes(int sum) { return kSeq + (uint32_t)sum + 4 * kPad + 16; }
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

// Where a pair's cells are: dlo rounded down to even (the diagonal below the
// band, if any, is masked), the band's indices [lo, hi).
struct TeamGeo {
  int L1, L2, dlo, lo, hi;
  int r0, j0;  // row and column of lane 0's first cell at double step 0
  int me;      // double step of the final cell
};
__device__ __forceinline__ TeamGeo team_geo(const LinPlan &P) {
  TeamGeo g;
  g.L1 = P.l1, g.L2 = P.l2;
  g.lo = P.dlo & 1;
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
};

// One double step.  cap: the final cell is in this one (0 even, 1 odd step):
// its registers go to `end`.
template <int MODE, int D>
__device__ __forceinline__ void team_step(TeamState<MODE, D> &S, const uint4 *cv, uint2 g, int lane,
                                          const DpK &K, int cap, uint32_t *end) {
  constexpr int NQ = D / 4;
  uint32_t W[2 * NQ];
#pragma unroll
  for (int v = 0; v < D / 8; ++v) {
    const uint4 x = cv[32 * v];
    W[4 * v] = x.x, W[4 * v + 1] = x.y, W[4 * v + 2] = x.z, W[4 * v + 3] = x.w;
  }
  const uint32_t one = (uint32_t)K.one;
#pragma unroll
  for (int q = NQ - 1; q > 0; --q) S.gd[q] = S.gd[q - 1];
  S.gd[0] = g.y;
  {
    uint32_t recv = __shfl_up_sync(kTFull, S.O[NQ - 1], 1);
    if (lane == 0) recv = kTInf2;
    const uint32_t lw = t_prmt(recv, S.O[NQ - 1], 0x5432);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      uint32_t x = __viaddmin_u16x2(S.E[q], W[q], t_mad(S.O[q], one, S.gd[q]));
      x = __viaddmin_u16x2(q ? S.O[q - 1] : lw, S.gi[q], x);
      if (MODE == kDpChoice) S.aE[q] = t_mad(S.aE[q], (uint32_t)K.four, x & 0x00030003u);
      S.E[q] = (x & S.kE[q]) | S.iE[q];
    }
  }
  if (cap == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) end[32 * q + lane] = S.E[q];
  }
#pragma unroll
  for (int q = 0; q + 1 < NQ; ++q) S.gi[q] = S.gi[q + 1];
  S.gi[NQ - 1] = g.x;
  {
    uint32_t recv = __shfl_down_sync(kTFull, S.E[0], 1);
    if (lane == 31) recv = kTInf2;
    const uint32_t rw = t_prmt(S.E[0], recv, 0x5432);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      uint32_t x = __viaddmin_u16x2(S.O[q], W[NQ + q], t_mad(S.E[q], one, S.gi[q]));
      x = __viaddmin_u16x2(q + 1 < NQ ? S.E[q + 1] : rw, S.gd[q], x);
      if (MODE == kDpChoice) S.aO[q] = t_mad(S.aO[q], (uint32_t)K.four, x & 0x00030003u);
      S.O[q] = (x & S.kO[q]) | S.iO[q];
    }
  }
  if (cap == 1) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) end[32 * q + lane] = S.O[q];
  }
}

// The traceback of one pair by one warp: tb_pair4_solo's walk (linear4.cu)
// over this layout's moves.  A diagonal run stays on one lane's words, so the
// window holds kTWalk chunks of that lane and its two neighbours.
template <int D>
__device__ __forceinline__ void team_walk(const LinTbArgs &A, const uint8_t *med, int id,
                                          const LinPlan &P, const uint32_t *dm, uint4 *win,
                                          const uint8_t *s1, const uint8_t *s2, int lane) {
  constexpr int NQ = D / 4, NV = D / 8;
  const TeamGeo g = team_geo(P);
  const int gap = A.gap;
  const int la = P.swap ? P.l2 : P.l1, lb = P.swap ? P.l1 : P.l2;
  const int64_t cap = slot_cap(la, lb);
  uint8_t *oa = A.out + A.out_off[id];
  uint8_t *ob = oa + cap, *ow = ob + cap, *om = ow + cap;
  const uint4 *dm4 = reinterpret_cast<const uint4 *>(dm);
  const uint32_t *win4 = reinterpret_cast<const uint32_t *>(win);
  const int nch = g.me / kTChunk + 1;
  const bool swaped = A.swaped < 0 ? !P.swap : (A.swaped != 0);
  int r = P.l1 - 1, j = P.l2 - 1;
  int n = 0, nm = 0, wlo = nch, wk = 0;  // window: chunks [wlo, wlo + kTWalk), lanes [wk, wk + 3)
  bool bad = false;
  while (r > 0 || (r == 0 && j >= 0)) {
    const int i = j - r - g.dlo;
    if (j < 0 || i < g.lo || i >= g.hi || n + 2 >= cap) {  // left the band: a bug
      bad = true;
      break;
    }
    const int k = i / D, c = (i % D) >> 1, par = i & 1;
    const int w = par * NQ + c % NQ, sh0 = 16 * (c / NQ);
    const int m0 = (r + j) >> 1;
    if (m0 / kTChunk < wlo || m0 / kTChunk >= wlo + kTWalk || k < wk || k >= wk + 3) {
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
    const int ri = r - lane, ji = j - lane, m = m0 - lane;
    uint32_t code = 4;
    if (ri >= 0 && ji >= 0 && n + lane + 2 < cap && m / kTChunk >= wlo) {
      const uint32_t x = win4[(((m / kTChunk - wlo) * NV + (w >> 2)) * 3 + (k - wk)) * 4 + (w & 3)];
      code = (x >> (2 * (7 - m % kTChunk) + sh0)) & 3u;
    }
    const uint32_t stop = __ballot_sync(kTFull, code != 0);
    const int f = stop ? __ffs(stop) - 1 : 32;  // lanes below f move diagonally
    const uint32_t cf = __shfl_sync(kTFull, code, f & 31);
    const bool step_f = f < 32 && cf != 4;
    const int move_f = step_f ? (((cf == 1u) == swaped) ? 1 : 2) : 0;
    const bool writes = lane < f || (lane == f && step_f);
    int md = gap;
    if (writes) {
      const bool dr = lane < f || move_f != 1, dj = lane < f || move_f != 2;
      const int cr = dr ? (int)s1[ri] : gap, cc = dj ? (int)s2[ji] : gap;
      const int ca = P.swap ? cc : cr, cb = P.swap ? cr : cc;
      md = med[(ca << 5) | cb];
      const int64_t pos = cap - 1 - (n + lane);
      oa[pos] = (uint8_t)ca;
      ob[pos] = (uint8_t)cb;
      ow[pos] = (uint8_t)md;
    }
    const bool keep = writes && md != gap;
    const uint32_t kb = __ballot_sync(kTFull, keep);
    if (keep) om[cap - 1 - (nm + __popc(kb & ((1u << lane) - 1u)))] = (uint8_t)md;
    n += f + (step_f ? 1 : 0);
    nm += __popc(kb);
    r -= f + ((step_f && move_f != 1) ? 1 : 0);
    j -= f + ((step_f && move_f != 2) ? 1 : 0);
  }
  if (lane == 0) {
    if (!bad) om[cap - 1 - nm] = (uint8_t)gap;  // ancestor_2 ends with the leading gap (algn.c:4140-4141)
    A.out_len[2 * id] = bad ? -1 : (int32_t)n;
    A.out_len[2 * id + 1] = bad ? -1 : (int32_t)(nm + 1);
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
  for (int e = tid; e < 33 * 33; e += kTThreads) {
    const int a = e / 33, b = e - 33 * a;
    tab[a * kTStride + b] =
        a < 32 && b < 32 ? (uint8_t)(sc * (A.tables->packed[(a << 5) | b] & 0xffffu)) : 0;
  }
  if (tid < 33) {
    gi_t[tid] = (uint16_t)((tid < 32 ? sc * (A.tables->packed[tid] >> 16) : 0) + rank_i);
    gd_t[tid] = (uint16_t)((tid < 32 ? sc * (A.tables->packed[(tid << 5) | A.gap] & 0xffffu) : 0) + rank_d);
  }
  if (MODE == kDpChoice)
    for (int i = tid; i < 1024; i += kTThreads) med[i] = A.tables->median[i];
  uint8_t *s1 = team_sm + Dm::kSeq + Dm::kPad, *s2 = s1 + g.L1 + 2 * Dm::kPad;
  for (int x = tid; x < g.L1 + 2 * Dm::kPad; x += kTThreads) {
    const int r = x - Dm::kPad;
    s1[r] = r >= 0 && r < g.L1 ? A.seq[P.s1_off + r] : (uint8_t)kTPadChar;
  }
  for (int x = tid; x < g.L2 + 2 * Dm::kPad; x += kTThreads) {
    const int j = x - Dm::kPad;
    s2[j] = j >= 0 && j < g.L2 ? A.seq[P.s2_off + j] : (uint8_t)kTPadChar;
  }
  __syncthreads();

  // a helper's share of chunk c: lane k, double step 8 c + (lane >> 2)
  auto produce = [&](int c) {
    const int k = 4 * (warp - 1) + (lane & 3), v = lane >> 2, m = kTChunk * c + v;
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
  } else {
    produce(0);
  }
  __syncthreads();
  for (int c = 0; c < nch; ++c) {
    if (warp != 0) {
      if (c + 1 < nch) produce(c + 1);
    } else {
      const uint8_t *slot = team_sm + (c & 1) * Dm::kSlot;
      if (c + 1 < nch) {
#pragma unroll
        for (int v = 0; v < kTChunk; ++v)
          team_step<MODE, D>(S, reinterpret_cast<const uint4 *>(slot + v * Dm::kStep) + lane,
                             reinterpret_cast<const uint2 *>(slot + v * Dm::kStep + NV * 512)[lane],
                             lane, A.k, -1, end);
      } else {
#pragma unroll 1
        for (int v = 0; v < kTChunk; ++v)
          team_step<MODE, D>(S, reinterpret_cast<const uint4 *>(slot + v * Dm::kStep) + lane,
                             reinterpret_cast<const uint2 *>(slot + v * Dm::kStep + NV * 512)[lane],
                             lane, A.k, v == g.me % kTChunk ? (fcell & 1) : -1, end);
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
  if (warp != 0) return;
  if (lane == 0) {
    const int cc = (fcell % D) >> 1;
    const uint32_t v = (end[32 * (cc % NQ) + fk] >> (16 * (cc / NQ))) & 0xFFFFu;
    A.cost[id] = ((int)v - (int)tab[s1[0] * kTStride + s2[0]]) / sc;
  }
  if (MODE == kDpChoice) {
    __syncwarp();
    team_walk<D>(A.tb, med, id, P, A.dm + id * A.dm_stride, reinterpret_cast<uint4 *>(team_sm), s1,
                 s2, lane);
  }
}

template <int MODE, int D>
int team_launch(const TeamArgs &A, int maxsum, cudaStream_t st) {
  static std::atomic<uint32_t> opted[64];
  const uint32_t sm = TeamDim<D>::bytes(maxsum);
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

// Diagonals per lane for bands up to maxwd (one more for the parity), 0 when
// the band or the sequences do not fit.
int lin_team_width(int maxwd, int maxsum) {
  const int d = maxwd + 1 <= 256 ? 8 : maxwd + 1 <= 512 ? 16 : maxwd + 1 <= 1024 ? 32 : 0;
  const uint32_t sm = d == 8 ? TeamDim<8>::bytes(maxsum) : d == 16 ? TeamDim<16>::bytes(maxsum)
                    : d == 32 ? TeamDim<32>::bytes(maxsum) : 0;
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
