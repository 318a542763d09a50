// Linear-gap banded DP by antidiagonals, in 16-bit halves, for large batches.
//
// Restates the recurrence of linear.cu (algn_fill_plane_2, algn.c:812-968) and
// backtrack_2d's choice (algn.c:3551-3666) for the batches whose values fit 16
// bits; k_lin_dp4 computes the same cells in rows.  There a warp takes a pair
// and its lanes, 7 steps apart, each meet strip switches and band edges at steps
// of their own, so nearly every step carries their selects and masks (about 60
// cycles for a lane's 4 cells).  Here the band lives in registers and nothing
// but the characters moves:
//   * 8, 16 or 32 lanes take a pair.  Lane k owns the D diagonals idx = D k ..
//     D k + D - 1, idx = j - i + off; the low half of E[q] is idx D k + 2q and
//     the high half D/2 above it, O[q] the odd ones between.  Step t = i + j
//     updates E (t even) from O or O from E: a cell's diagonal predecessor is
//     its own old value, the left one the diagonal below and the upper one the
//     diagonal above, so one shuffle a step serves the lane's edge;
//   * off is even, so that E and O are the even and odd steps; the diagonals
//     below the band (idx 0, or 0 and 1) and above it are forced to infinity by
//     a LOP3 that also clears the rank bits;
//   * a cell's cost is one byte of shared memory: the table is there 32 times, a
//     word of each copy in the lane's own bank (a single copy, two cells a lookup,
//     met 3.7 lanes in a bank on sequences with 5 % ambiguity codes and was no
//     faster than k_lin_dp4);
//   * rows and columns are turned into (gap cost, table offset) once per pair
//     and pass its lanes through a ring in shared memory, D/2 at a time: lane k
//     reads the chunk k behind the first lane's.
// Outside the matrix the codes are 0 (no code of a batch: the plan refuses 0),
// whose costs here are 0, so infinity stays infinity.
//
// kDpChoice keeps values x 4 with the move's rank in the low bits as k_lin_dp4
// does; a direction word holds a register's two cells over a block of four to
// seven double steps, the pair's words are [block][lane][register].
//
// Bound: instruction issue (81-90 % of the slots; for two cells 2 address adds, 2
// lookups, a multiply-add that joins them, an add, 2 add-mins and a LOP3, with
// directions 2 rank multiply-adds).  Measured against k_lin_dp4, whose lanes work
// 7 steps apart and so meet strips and edges at steps of their own (60 cycles for
// four cells): the costs of 154,296 pairs of 1,500 bp 29.5 and 18.4 ms; 65,536
// pairs of 100-5,000 bp with their walk 29.1 and 21.4 ms.
#include <algorithm>
#include <atomic>
#include <cuda_runtime.h>
#include <cstdint>
#include "poyd_internal.h"
#include "linear_kernels.cuh"

namespace poyd {
namespace {

constexpr unsigned kGFull = 0xffffffffu;
constexpr unsigned kGInf2 = 0xC000C000u;
constexpr unsigned kGRk = 0x00030003u;
// Warps of a block (one an SM).  With directions the registers of twelve, more
// lookups in flight a warp, are worth more than four warps: the 65,536-pair batch
// of 100-5,000 bp 18.9 against 19.6 ms; without, 38,912 pairs of 1,500 bp 5.4 ms
// with sixteen and 5.7 with twelve.
template <bool BT>
__host__ __device__ constexpr int diag_warps() {
  return BT ? 12 : 16;
}
constexpr int kGMaxC = 14;  // widest class: 28 diagonals a lane
constexpr int kGRow = 8 * 128;  // bytes of a row code's part of the table

template <bool BT>
struct DiagPairSmem {
  uint2 ring[diag_warps<BT>()][2][32 * (kGMaxC + 1)];  // rows, columns: gap cost, table offset
  uint2 stage[BT ? diag_warps<BT>() : 1][32 * kGMaxC / 2];  // direction words on their way out
  uint8_t cost[32 * kGRow];   // [row code][column code / 4][lane][column code % 4]
  uint16_t del[32], ins[32];  // sc * cost[c][gap], sc * cost[gap][c]
};

__device__ __forceinline__ unsigned g_prmt(unsigned a, unsigned b, unsigned s) {
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}
__device__ __forceinline__ unsigned g_mad(unsigned a, unsigned b, unsigned c) {
  unsigned d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Shared loads and stores by 32-bit address.  The table does not change.
__device__ __forceinline__ unsigned g_table(unsigned a) {
  unsigned v;
  asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 g_lds(unsigned a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void g_sts(unsigned a, unsigned x, unsigned y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}

__device__ __forceinline__ void g_near(unsigned sink, const void *p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sink), "l"(p) : "memory");
}

// Byte offsets in the table, for every lane a word in its own bank.
__device__ __forceinline__ unsigned row_offset(int c) { return (unsigned)c * kGRow; }
__device__ __forceinline__ unsigned col_offset(int c) { return ((unsigned)c >> 2) * 128 + (c & 3); }

template <bool BT, int D>
struct LinDiagState {
  static constexpr int NQ = D / 4, C = D / 2;
  unsigned h[2][NQ];          // values: 0 even, 1 odd
  unsigned rv[NQ], cv[NQ];    // gap costs of the cells' rows and columns
  unsigned mask[2][NQ];       // halves forced to infinity; the rank bits
  unsigned arow[C], bcol[C + 1];  // table offsets of the cells' rows and columns
  unsigned acc[2][BT ? NQ : 1];
};

// What one lane knows of its pair.
struct LinDiagLane {
  const uint8_t *s1, *s2;
  int l1, l2, k, lanes, base;
  unsigned rank_d, rank_i;
  unsigned rows, cols;  // the group's rings
  unsigned tab;         // the lane's words of the cost table
  unsigned stage;       // the group's direction words of eight double steps
  int below, above;
  int ch[2][2];  // characters of the next chunk's places: row, column
};

template <int D>
__device__ __forceinline__ void ld_row(unsigned (&rv)[D / 4], unsigned (&arow)[D / 2], uint2 r, unsigned tab) {
  constexpr int NQ = D / 4;
  const unsigned last = rv[NQ - 1];
#pragma unroll
  for (int q = NQ - 1; q > 0; --q) rv[q] = rv[q - 1];
  rv[0] = g_prmt(r.x, last, 0x5410);
#pragma unroll
  for (int c = D / 2 - 1; c > 0; --c) arow[c] = arow[c - 1];
  arow[0] = r.y + tab;
}
template <int D>
__device__ __forceinline__ void ld_col(unsigned (&cv)[D / 4], unsigned x) {
  constexpr int NQ = D / 4;
  const unsigned first = cv[0];
#pragma unroll
  for (int q = 0; q + 1 < NQ; ++q) cv[q] = cv[q + 1];
  cv[NQ - 1] = g_prmt(first, x, 0x5432);
}
template <int D>
__device__ __forceinline__ void ld_char(unsigned (&bcol)[D / 2 + 1], unsigned y) {
#pragma unroll
  for (int c = 0; c < D / 2; ++c) bcol[c] = bcol[c + 1];
  bcol[D / 2] = y;
}

// The characters of row and column chunk n (rows base + C n .., columns
// C lanes - base + C n ..), a lane a place (two where C exceeds eight lanes).
template <int D>
__device__ __forceinline__ void ld_chars(LinDiagLane &L, int n) {
  constexpr int C = D / 2;
#pragma unroll
  for (int e = 0; e < (C > 8 ? 2 : 1); ++e) {
    if (e && L.lanes > 8) break;
    const int x = L.k + 8 * e;
    const int row = L.base + C * n + x, col = C * L.lanes - L.base + C * n + x;
    const bool on = x < C;
    L.ch[e][0] = on && row >= 0 && row < L.l1 ? (int)__ldg(L.s1 + row) : 0;
    L.ch[e][1] = on && col >= 0 && col < L.l2 ? (int)__ldg(L.s2 + col) : 0;
  }
}
// Chunk n into the rings, from the characters read a chunk ago.
template <bool BT, int D>
__device__ __forceinline__ void ld_produce(LinDiagLane &L, const DiagPairSmem<BT> &sm, int n) {
  constexpr int C = D / 2;
  __syncwarp();  // the places written over have been read
#pragma unroll
  for (int e = 0; e < (C > 8 ? 2 : 1); ++e) {
    if (e && L.lanes > 8) break;
    const int x = L.k + 8 * e;
    if (x < C) {
      const int row = L.base + C * n + x, col = C * L.lanes - L.base + C * n + x;
      const int at = (n & (L.lanes - 1)) * (C | 1) + x;
      const int a = L.ch[e][0], b = L.ch[e][1];
      const bool in1 = row >= 0 && row < L.l1, in2 = col >= 0 && col < L.l2;
      // row 0 and column 0 have no diagonal predecessor
      g_sts(L.rows + 8 * at, in1 ? sm.del[a] + L.rank_d : 0u, row_offset(row > 0 ? a : 0));
      g_sts(L.cols + 8 * at, in2 ? sm.ins[b] + L.rank_i : 0u, col_offset(col > 0 ? b : 0));
    }
  }
  ld_chars<D>(L, n + 1);
  __syncwarp();
}

// The step of parity X.
template <bool BT, int D, int X>
__device__ __forceinline__ void ld_step(LinDiagState<BT, D> &S, int src, unsigned mul, const DpK &K) {
  constexpr int NQ = D / 4, Y = 1 - X;
  const unsigned one = (unsigned)K.one;
  const unsigned out = S.h[Y][X == 0 ? NQ - 1 : 0];
  const unsigned nb = __shfl_sync(kGFull, out, src);
  const unsigned edge = X == 0 ? g_prmt(nb, out, 0x5432) : g_prmt(out, nb, 0x5432);
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const unsigned left = X == 0 ? (q ? S.h[Y][q ? q - 1 : 0] : edge) : S.h[Y][q];
    const unsigned up = X == 0 ? S.h[Y][q] : (q + 1 < NQ ? S.h[Y][q + 1 < NQ ? q + 1 : 0] : edge);
    const unsigned cd = g_mad(g_table(g_mad(S.arow[q + NQ], one, S.bcol[q + NQ + X])),
                              (unsigned)K.k64, g_table(g_mad(S.arow[q], one, S.bcol[q + X])));
    unsigned v = __viaddmin_u16x2(S.h[X][q], cd, g_mad(left, one, S.cv[q]));
    v = __viaddmin_u16x2(up, S.rv[q], v);
    const unsigned m = S.mask[X][q];
    const unsigned c = (v & ~m) | (kGInf2 & m);
    if (BT) {
      // the forced low half of register 0 would borrow from the high one
      const unsigned r = q == 0 ? v & kGRk : g_mad(c, (unsigned)K.m1, v);
      S.acc[X][q] = g_mad(S.acc[X][q], mul, r);
    }
    S.h[X][q] = c;
  }
}

// Double step m, the u-th of its block, whose first is at rows and cols in the
// rings.
// CHECK: some pair's final cell may be in it.
template <bool BT, int D, bool CHECK>
__device__ __forceinline__ void ld_double(LinDiagState<BT, D> &S, const LinDiagLane &L,
                                          unsigned rows,
                                          unsigned cols, int u, int m, int fin, int fq,
                                          unsigned &res, const DpK &K) {
  constexpr int NQ = D / 4;
  ld_row<D>(S.rv, S.arow, g_lds(rows + 8 * u), L.tab);
  const uint2 r = g_lds(cols + 8 * u);
  ld_char<D>(S.bcol, r.y);
  const unsigned mul = BT && u ? (unsigned)K.four : 0u;
  ld_step<BT, D, 0>(S, L.below, mul, K);
  if (CHECK && 2 * m == fin) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) res = q == fq ? S.h[0][q] : res;
  }
  ld_col<D>(S.cv, r.x);
  ld_step<BT, D, 1>(S, L.above, mul, K);
  if (CHECK && 2 * m + 1 == fin) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) res = q == fq ? S.h[1][q] : res;
  }
}

// The direction words of a block of double steps, gathered so that a lane's
// words lie side by side (the walk's next words) and the group's in one run.
template <bool BT, int D>
__device__ __forceinline__ void ld_flush(const LinDiagState<BT, D> &S, const LinDiagLane &L,
                                         uint2 *dw, int block, int blocks) {
  constexpr int NQ = D / 4;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    g_sts(L.stage + 8 * (L.k * NQ + q), S.acc[0][BT ? q : 0], S.acc[1][BT ? q : 0]);
  __syncwarp();
  const bool mine = block < blocks;
#pragma unroll
  for (int v = 0; v < NQ; ++v) {
    const uint2 x = g_lds(L.stage + 8 * (v * L.lanes + L.k));
    if (mine) dw[(block * NQ + v) * L.lanes] = x;
  }
  __syncwarp();
}

// A task: the pairs of positions p .. p + 32 / lanes - 1 below `end`.
template <bool BT, int D>
__device__ __forceinline__ void ld_task(const LinDiagArgs &A, const DiagPairSmem<BT> &sm, uint2 *ring,
                                        uint2 *stage, int p, int end, int lanes, int lane) {
  constexpr int NQ = D / 4, C = D / 2, U = lin_diag_block(D);
  constexpr int sc = BT ? 4 : 1;
  LinDiagLane L;
  const int grp = lane / lanes;
  L.lanes = lanes;
  L.k = lane & (lanes - 1);
  const int id = p + grp < end ? A.order[p + grp] : -1;
  L.s1 = L.s2 = A.seq;
  L.l1 = L.l2 = 0;
  L.base = 0;
  L.rank_d = L.rank_i = 0;
  int top = 0, low = 1;  // the band's idx: low .. top - 1
  uint2 *dw = nullptr;
  bool has = false;
  if (id >= 0) {
    const LinPlan P = A.plans[id];
    if (P.empty) {
      if (L.k == 0) A.cost[id] = 0;
    } else {
      has = true;
      L.l1 = P.l1, L.l2 = P.l2;
      L.s1 += P.s1_off, L.s2 += P.s2_off;
      L.base = lin_diag_off(P.dlo) / 2;
      low = P.dlo + 2 * L.base;
      top = low + P.wd;
      // backtrack priority (algn.c:3605-3666): insert before delete when swaped
      if (BT) {
        L.rank_i = P.swap ? 2 : 1;
        L.rank_d = 3 - L.rank_i;
        dw = reinterpret_cast<uint2 *>(A.dm + A.dm_off[id]) + L.k;
      }
    }
  }
  const int fin = has ? L.l1 + L.l2 - 2 : -1;  // the final cell's step
  const int blocks = BT && has ? (fin >> 1) / U + 1 : 0;
  const int last = __reduce_max_sync(kGFull, fin >> 1);
  const int fidx = L.l2 - L.l1 + 2 * L.base, fk = fidx / D, fc = fidx % D >> 1;
  LinDiagState<BT, D> S;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      S.h[x][q] = kGInf2;
      unsigned m = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int idx = D * L.k + 2 * (q + h * NQ) + x;
        if (idx < low || idx >= top) m |= 0xFFFFu << (16 * h);
        // cell (0, 0) is 0: its diagonal predecessor is, and costs nothing
        if (has && idx == 2 * L.base) S.h[x][q] &= ~(0xFFFFu << (16 * h));
      }
      S.mask[x][q] = BT ? m | kGRk : m;
      if (BT) S.acc[x][q] = 0;
    }
#pragma unroll
  for (int q = 0; q < NQ; ++q) S.rv[q] = S.cv[q] = 0;
  L.tab = (unsigned)__cvta_generic_to_shared(sm.cost) + 4 * lane;
  const unsigned none = row_offset(0) + L.tab;
#pragma unroll
  for (int c = 0; c < C; ++c) S.arow[c] = none;
#pragma unroll
  for (int c = 0; c <= C; ++c) S.bcol[c] = col_offset(0);
  // a chunk takes an odd number of places: the lanes' reads meet no bank twice
  L.rows = (unsigned)__cvta_generic_to_shared(ring) + 8 * grp * lanes * (C | 1);
  L.cols = L.rows + 8 * 32 * (kGMaxC + 1);
  L.stage = (unsigned)__cvta_generic_to_shared(stage) + 8 * grp * lanes * NQ;
  L.below = (lane - L.k) | ((L.k - 1) & (lanes - 1));
  L.above = (lane - L.k) | ((L.k + 1) & (lanes - 1));
  ld_chars<D>(L, -lanes);
#pragma unroll 1
  for (int n = -lanes; n < 0; ++n) ld_produce<BT, D>(L, sm, n);
  auto rows_at = [&](int n) { return L.rows + 8 * ((n - L.k) & (lanes - 1)) * (C | 1); };
  auto cols_at = [&](int n) { return L.cols + 8 * ((n + 1 + L.k) & (lanes - 1)) * (C | 1); };
  {
    const unsigned r = rows_at(-1), c = cols_at(-1);
#pragma unroll 1
    for (int u = 0; u < C; ++u) {  // the registers' first rows and columns
      ld_row<D>(S.rv, S.arow, g_lds(r + 8 * u), L.tab);
      const uint2 y = g_lds(c + 8 * u);
      ld_char<D>(S.bcol, y.y);
      ld_col<D>(S.cv, y.x);
    }
  }
  unsigned res = 0;
  int n = 0;
#pragma unroll 1
  for (int m = 0; m <= last; m += C, ++n) {
    ld_produce<BT, D>(L, sm, n);
    const unsigned r = rows_at(n), c = cols_at(n);
    const bool check = __any_sync(kGFull, fin >= 2 * m && fin < 2 * (m + C));
#pragma unroll 1
    for (int e = 0; e < C; e += U) {
      if (check) {
#pragma unroll 1
        for (int u = 0; u < U; ++u)
          ld_double<BT, D, true>(S, L, r + 8 * e, c + 8 * e, u, m + e + u, fin, fc % NQ, res, A.k);
      } else {
        // the registers' places turn by one a double step: C of them unrolled
        // bring them back without moves, half of them with few; more code would
        // not stay in the instruction cache
#pragma unroll
        for (int u = 0; u < U; ++u)
          ld_double<BT, D, false>(S, L, r + 8 * e, c + 8 * e, u, m + e + u, fin, fc % NQ, res, A.k);
      }
      if (BT) ld_flush<BT, D>(S, L, dw, (m + e) / U, blocks);
    }
  }
  res = __shfl_sync(kGFull, res, (lane - L.k) + (has ? fk : 0));
  if (has && L.k == 0) A.cost[id] = (int)(res >> (16 * (fc / NQ)) & 0xFFFFu) / sc;
  __syncwarp();
}

template <bool BT>
__global__ void __launch_bounds__(diag_warps<BT>() * 32, 1) k_lin_diag(const __grid_constant__ LinDiagArgs A) {
  extern __shared__ __align__(16) uint8_t lin_diag_sm[];
  DiagPairSmem<BT> &sm = *reinterpret_cast<DiagPairSmem<BT> *>(lin_diag_sm);
  constexpr int sc = BT ? 4 : 1;
  for (int e = threadIdx.x >> 5; e < 256; e += diag_warps<BT>()) {  // row code e / 8, four column codes
    unsigned w = 0;
    for (int x = 0; x < 4; ++x)
      if (e >= 8 && 4 * (e & 7) + x) w |= (sc * (A.tables->packed[4 * e + x] & 0xffffu)) << (8 * x);
    reinterpret_cast<unsigned *>(sm.cost)[32 * e + (threadIdx.x & 31)] = w;
  }
  if (threadIdx.x < 32) {
    sm.del[threadIdx.x] = (uint16_t)(sc * (A.tables->packed[(threadIdx.x << 5) | 16] & 0xffffu));
    sm.ins[threadIdx.x] = (uint16_t)(sc * (A.tables->packed[threadIdx.x] >> 16));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint2 *ring = sm.ring[threadIdx.x >> 5][0], *stage = sm.stage[BT ? threadIdx.x >> 5 : 0];
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(A.counter, 1);
    t = __shfl_sync(kGFull, t, 0);
    if (t >= A.tasks[kLinDiagClasses]) break;
    int c = 0;
    while (t >= A.tasks[c + 1]) ++c;
    const int lanes = lin_diag_class(c).lanes, width = lin_diag_class(c).width;
    const int per = 32 / lanes, end = A.base[c + 1];
    const int p = A.base[c] + (t - A.tasks[c]) * per;
    if (width == 8) ld_task<BT, 8>(A, sm, ring, stage, p, end, lanes, lane);
    else if (width == 12) ld_task<BT, 12>(A, sm, ring, stage, p, end, lanes, lane);
    else if (width == 16) ld_task<BT, 16>(A, sm, ring, stage, p, end, lanes, lane);
    else if (width == 20) ld_task<BT, 20>(A, sm, ring, stage, p, end, lanes, lane);
    else if (width == 24) ld_task<BT, 24>(A, sm, ring, stage, p, end, lanes, lane);
    else ld_task<BT, 28>(A, sm, ring, stage, p, end, lanes, lane);
  }
}

// ---------------------------------------------------------------------------
// Traceback (backtrack_2d, algn.c:3551-3666) and medians (ancestor_2,
// algn.c:4126-4147; median_2_with_gaps, algn.c:4011-4024) in two kernels: a
// thread follows a pair's path, a run of diagonal moves and the next other one a
// step, and leaves its moves as 2-bit ranks, 16 a word; then a warp a pair writes the sequences, a lane a column.
// (Inside k_lin_diag, by the warp that completes 32 pairs or by the pair's own,
// the walk shared the instruction cache with the sweep and waited for memory on
// every step: 2.7 ms more for the 65,536-pair batch, in the best of five forms.)
// ---------------------------------------------------------------------------
struct DiagPair {
  int id, lanes, width;
  int64_t words;
};
// The pair of position p (of those from A.base[0]).
__device__ __forceinline__ DiagPair diag_pair(const LinDiagArgs &A, int p) {
  int c = 0;
  while (p >= A.base[c + 1]) ++c;
  const int id = A.order[p];
  return DiagPair{id, lin_diag_class(c).lanes, lin_diag_class(c).width,
                  lin_diag_words(c, A.plans[id].l1 + A.plans[id].l2)};
}

// The moves go into the words of the pair's matrix that the path has passed, from
// the end (16 columns take at least eight double steps, more than a block).
// Bound: the memory latency of a step.
__global__ void __launch_bounds__(64) k_diag_path(const __grid_constant__ LinDiagArgs A, int per) {
  const int lane = threadIdx.x & 31;
  const int p = A.base[0] + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per + lane;
  if (lane >= per || p >= A.base[kLinDiagClasses]) return;
  const DiagPair D = diag_pair(A, p);
  const LinPlan P = A.plans[D.id];
  if (P.empty) return;
  uint32_t *dm = A.dm + A.dm_off[D.id], *path = dm + D.words;
  const int64_t cap = slot_cap(P.l1, P.l2);
  const int off = lin_diag_off(P.dlo), low = P.dlo + off;
  const int width = D.width, NQ = width / 4, stride = D.lanes * 2 * NQ;  // words of a block
  const unsigned U = lin_diag_block(width), iw = 0xFFFFFFFFu / width + 1, iu = 0xFFFFFFFFu / U + 1;
  const unsigned first = P.swap ? 2u : 1u;  // the rank of an insert
  int r = P.l1 - 1, j = P.l2 - 1;
  int n = 0, key = -1;
  bool bad = false;
  uint32_t cur = 0, moves = 0;
  int last = -1;
  __shared__ uint32_t sinks[64];
  const unsigned sink = (unsigned)__cvta_generic_to_shared(sinks + threadIdx.x);
  while (r >= 0 && (r > 0 || j >= 0)) {
    const int idx = j - r + off;
    if (j < 0 || (unsigned)(idx - low) >= (unsigned)P.wd || n + 2 >= cap) {  // left the band: a bug
      bad = true;
      break;
    }
    const int k = (int)__umulhi((unsigned)idx, iw), m = (r + j) >> 1;
    const int block = (int)__umulhi((unsigned)m, iu);
    int c = (idx - k * width) >> 1, sh = 2 * ((block + 1) * (int)U - 1 - m);
    if (c >= NQ) c -= NQ, sh += 16;
    const int at = block * stride + k * 2 * NQ + 2 * c + (idx & 1);
    if (at != key) {
      cur = dm[key = at];
      // the lane's words three blocks on, into the L1 cache
      const int far = (block - 3) * stride + k * 2 * NQ;
      if (block >= 3 && block != last) {
        g_near(sink, dm + far);
        g_near(sink, dm + far + 2 * NQ - 1);
      }
      last = block;
    }
    // the diagonal moves that the word shows, then the other one behind them
    const int left = m - block * (int)U + 1;  // steps of the word
    const uint32_t code = cur >> sh;
    int f = (__ffs((int)(code | 1u << (2 * left))) - 1) >> 1;
    f = min(f, min(min(r, j) + 1, (int)min(cap - 2 - n, (int64_t)left)));
    if ((n ^ (n + f)) & ~15) {
      path[-1 - (n >> 4)] = moves;
      moves = 0;
    }
    n += f;
    r -= f;
    j -= f;
    const unsigned rank = f < left ? (code >> (2 * f)) & 3u : 0u;
    if (rank && n + 2 < cap) {
      moves |= rank << (2 * (n & 15));
      if ((++n & 15) == 0) {
        path[-(n >> 4)] = moves;
        moves = 0;
      }
      r -= rank != first;
      j -= rank == first;
    } else if (f == 0) {  // no move of any kind: a bug
      bad = true;
      break;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (n & 15) path[-1 - (n >> 4)] = moves;
  A.tb.out_len[2 * D.id] = bad ? -1 : n;
}

// Bound: the bytes written (670 MB for the 65,536-pair batch).
__global__ void __launch_bounds__(128) k_diag_write(const __grid_constant__ LinDiagArgs A) {
  __shared__ uint8_t med[1024];
  for (int e = threadIdx.x; e < 1024; e += blockDim.x) med[e] = A.tables->median[e];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int p = A.base[0] + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (p >= A.base[kLinDiagClasses]) return;
  const DiagPair D = diag_pair(A, p);
  const LinPlan P = A.plans[D.id];
  const int gap = A.tb.gap;
  const int la = P.swap ? P.l2 : P.l1, lb = P.swap ? P.l1 : P.l2;
  const int64_t cap = slot_cap(la, lb);
  uint8_t *oa = A.tb.out + A.tb.out_off[D.id];
  uint8_t *ob = oa + cap, *ow = ob + cap, *om = ow + cap;
  const uint8_t *__restrict__ s1 = A.seq + P.s1_off;
  const uint8_t *__restrict__ s2 = A.seq + P.s2_off;
  if (P.empty) {
    // DOS.median: the non-empty (or second) sequence is the median
    const bool a_empty = P.empty == 1;
    const uint8_t *src = (a_empty != (bool)P.swap) ? s2 : s1;
    const int len = a_empty ? lb : la;
    for (int i = lane; i < len; i += 32) om[cap - len + i] = src[i];
    if (lane == 0) {
      A.tb.out_len[2 * D.id] = 0;
      A.tb.out_len[2 * D.id + 1] = len;
    }
    return;
  }
  const int n = A.tb.out_len[2 * D.id];
  const uint32_t *path = A.dm + A.dm_off[D.id] + D.words;
  const unsigned first = P.swap ? 2u : 1u, lt = (1u << lane) - 1u;
  uint8_t *row = (P.swap ? ob : oa) + cap - 1, *col = (P.swap ? oa : ob) + cap - 1;
  int r = P.l1 - 1, j = P.l2 - 1, nm = 0;
  constexpr int E = 4;  // 32 columns each, their loads together
  for (int v = 0; v < n; v += 32 * E) {
    unsigned code[E];
    int cr[E], cc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = v + 32 * e + lane;
      code[e] = x < n ? path[-1 - (x >> 4)] >> (2 * (lane & 15)) & 3u : 3u;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const bool dr = code[e] != 3 && code[e] != first, dj = code[e] == 0 || code[e] == first;
      const unsigned rb = __ballot_sync(kGFull, dr), jb = __ballot_sync(kGFull, dj);
      cr[e] = dr ? (int)__ldg(s1 + r - __popc(rb & lt)) : gap;
      cc[e] = dj ? (int)__ldg(s2 + j - __popc(jb & lt)) : gap;
      r -= __popc(rb);
      j -= __popc(jb);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = v + 32 * e + lane;
      const int md = med[P.swap ? (cc[e] << 5) | cr[e] : (cr[e] << 5) | cc[e]];
      const bool in = x < n;
      const unsigned kb = __ballot_sync(kGFull, in && md != gap);
      if (in) {
        row[-x] = (uint8_t)cr[e];
        col[-x] = (uint8_t)cc[e];
        ow[cap - 1 - x] = (uint8_t)md;
        if (md != gap) om[cap - 1 - nm - __popc(kb & lt)] = (uint8_t)md;
      }
      nm += __popc(kb);
    }
  }
  if (lane == 0) {
    // ancestor_2 ends with the leading gap (algn.c:4140-4141)
    if (n >= 0) om[cap - 1 - nm] = (uint8_t)gap;
    A.tb.out_len[2 * D.id + 1] = n < 0 ? -1 : nm + 1;
  }
}

// ---------------------------------------------------------------------------
// Order: by class (widest band first, the pairs no class holds last), within it
// longest first by log2 buckets of l1 + l2.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int diag_key(const LinPlan &P, int min_lanes, int *c) {
  *c = lin_diag_class_of(P.dlo, P.wd, min_lanes);
  const unsigned sum = (unsigned)(P.l1 + P.l2) + 1;
  const int lg = 31 - __clz((int)sum);
  const int frac = lg >= 3 ? (sum >> (lg - 3)) & 7 : (sum << (3 - lg)) & 7;
  return *c * kLinDiagBuckets + kLinDiagBuckets - 1 - min(lg * 8 + frac, kLinDiagBuckets - 1);
}

// A warp's pairs of one bucket are counted at once: a batch's pairs share few.
__device__ __forceinline__ int bucket_add(int *hist, int key, bool ok, int lane) {
  const unsigned same = __match_any_sync(kGFull, ok ? key : -1);
  const int leader = __ffs(same) - 1;
  int at = 0;
  if (ok && lane == leader) at = atomicAdd(hist + key, __popc(same));
  at = __shfl_sync(kGFull, at, leader);
  return at + __popc(same & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(128) k_diag_count(int n, int min_lanes, bool bt,
                                                    const LinPlan *plans, const int64_t *dm_words,
                                                    int64_t *dm_off, LinDiagOrder *os) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool ok = id < n;
  int wd = 0, key = -1;
  unsigned long long w = 0, w4 = 0;
  if (ok) {
    const LinPlan P = plans[id];
    int c;
    key = diag_key(P, min_lanes, &c);
    wd = P.wd;
    w4 = (unsigned long long)dm_words[id];
    w = c < kLinDiagClasses ? (bt ? lin_diag_words(c, P.l1 + P.l2) : 0) : w4;
  }
  bucket_add(os->hist, key, ok, lane);
  unsigned long long incl = w, sum4 = w4;
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long x = __shfl_up_sync(kGFull, incl, d);
    if (lane >= d) incl += x;
    sum4 += __shfl_xor_sync(kGFull, sum4, d);
  }
  unsigned long long base = 0;
  if (lane == 31) base = atomicAdd(&os->total, incl);
  base = __shfl_sync(kGFull, base, 31);
  if (ok) dm_off[id] = (int64_t)(base + incl - w);
  wd = __reduce_max_sync(kGFull, wd);
  if (lane == 0) {
    atomicAdd(&os->total4, sum4);
    atomicMax(&os->maxwd, wd);
  }
}

__global__ void __launch_bounds__(1024) k_diag_scan(LinDiagOrder *os) {
  constexpr int kAll = (kLinDiagClasses + 1) * kLinDiagBuckets, kPer = (kAll + 1023) / 1024;
  __shared__ int part[32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int v[kPer], sum = 0;
  for (int e = 0; e < kPer; ++e) {
    v[e] = t * kPer + e < kAll ? os->hist[t * kPer + e] : 0;
    sum += v[e];
  }
  int incl = sum;
  for (int d = 1; d < 32; d <<= 1) {
    const int x = __shfl_up_sync(kGFull, incl, d);
    if (lane >= d) incl += x;
  }
  if (lane == 31) part[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int p = part[lane];
    for (int d = 1; d < 32; d <<= 1) {
      const int x = __shfl_up_sync(kGFull, p, d);
      if (lane >= d) p += x;
    }
    part[lane] = p;
  }
  __syncthreads();
  int at = (warp ? part[warp - 1] : 0) + incl - sum;
  for (int e = 0; e < kPer; ++e) {
    const int x = t * kPer + e;
    if (x >= kAll) break;
    os->hist[x] = at;  // now the scatter cursor
    if (x % kLinDiagBuckets == 0) os->base[x / kLinDiagBuckets] = at;
    at += v[e];
  }
}

__global__ void __launch_bounds__(128) k_diag_scatter(int n, int min_lanes, const LinPlan *plans,
                                                      LinDiagOrder *os, int32_t *order) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  const bool ok = id < n;
  int c, key = -1;
  if (ok) key = diag_key(plans[id], min_lanes, &c);
  const int at = bucket_add(os->hist, key, ok, threadIdx.x & 31);
  if (ok) order[at] = id;
}

__global__ void k_diag_flags(int *done, int b0, int b1) {
  const int b = b0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (b < b1) *(volatile int *)(done + b) = 1;
}

template <bool BT>
int diag_blocks() {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int c = cache[dev & 63].load();
  if (!c) {
    cudaFuncSetAttribute(k_lin_diag<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(DiagPairSmem<BT>));
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    cache[dev & 63].store(c = std::max(c, 1));
  }
  return c;
}

}  // namespace

// Fewer lanes a pair waste less of the band's width and of a double step's fixed
// part; more, while warps would idle.  (Alignments come here from more pairs than
// warps on: theirs take 32 lanes for bands that 16 do not hold alone.)
int lin_diag_min_lanes(int n, int sms, bool bt) {
  const int warps = sms * (bt ? diag_warps<true>() : diag_warps<false>());
  return !bt && n <= warps ? 32 : n <= 2 * warps ? 16 : 8;
}

void launch_lin_diag_order(int n, int min_lanes, bool bt, const LinPlan *plans,
                           const int64_t *dm_words, int64_t *dm_off, LinDiagOrder *os,
                           int32_t *order, cudaStream_t st) {
  const unsigned blocks = (unsigned)(((int64_t)n + 127) / 128);
  k_diag_count<<<blocks, 128, 0, st>>>(n, min_lanes, bt, plans, dm_words, dm_off, os);
  k_diag_scan<<<1, 1024, 0, st>>>(os);
  k_diag_scatter<<<blocks, 128, 0, st>>>(n, min_lanes, plans, os, order);
}

int launch_lin_diag(LinDiagArgs &A, bool bt, const int *base, cudaStream_t st) {
  A.tasks[0] = 0;
  for (int c = 0; c < kLinDiagClasses; ++c) {
    const int per = 32 / lin_diag_class(c).lanes;
    A.base[c] = base[c];
    A.tasks[c + 1] = A.tasks[c] + (base[c + 1] - base[c] + per - 1) / per;
  }
  A.base[kLinDiagClasses] = base[kLinDiagClasses];
  const int tasks = A.tasks[kLinDiagClasses];
  const int blocks = std::min(bt ? diag_blocks<true>() : diag_blocks<false>(), tasks);
  if (bt) k_lin_diag<true><<<blocks, 32 * diag_warps<true>(), sizeof(DiagPairSmem<true>), st>>>(A);
  else k_lin_diag<false><<<blocks, 32 * diag_warps<false>(), sizeof(DiagPairSmem<false>), st>>>(A);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "k_lin_diag") : POYD_OK;
}

int launch_lin_diag_walk(const LinDiagArgs &A, cudaStream_t st) {
  const unsigned n = (unsigned)(A.base[kLinDiagClasses] - A.base[0]);
  // four pairs a warp: the fewer, the fewer wait for another's memory (32: 1.5 ms
  // for 608 pairs of 5,000 bp, 16: 0.58, 8: 0.50, 4: 0.45, their writing included)
  const int per = 4;
  k_diag_path<<<(n + 2 * per - 1) / (2 * per), 64, 0, st>>>(A, per);
  k_diag_write<<<(n + 3) / 4, 128, 0, st>>>(A);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "k_diag_write") : POYD_OK;
}

int launch_lin_diag_flags(int *done, int b0, int b1, cudaStream_t st) {
  k_diag_flags<<<(b1 - b0 + 255) / 256, 256, 0, st>>>(done, b0, b1);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "k_diag_flags") : POYD_OK;
}

}  // namespace poyd
