// Affine-gap banded DP by antidiagonals, in 16-bit halves.
//
// Restates the fills and the traceback of affine.cu (algn_fill_plane_3_aff and
// _nobt, algn.c:1740-2548; backtrace_affine, algn.c:1983-2097) for batches
// whose values provably fit 16 bits; k_aff_dp2 computes the same cells in rows.
// There a lane's cell needs four shuffled states, a column record and a
// boundary test per cell (82 instructions a cell); here the band lives in
// registers:
//   * eight lanes take a pair, four pairs a warp (16 or 32 lanes where the band is
//     wider than 128 or 256, 16 in small batches with directions).  Lane k owns the D diagonals
//     idx = D k .. D k + D - 1 of the band (idx = d + 40, d = j - i), each
//     register two cells of one parity: E[q] idx 2q in the low half and 2q + D/2
//     in the high half, O[q] the odd ones above.  Step t updates the cells i + j
//     = t, even steps E from O and odd steps O from E: a cell's diagonal
//     predecessors are its own registers, the left one (EH, CB) the diagonal
//     below, the upper one (EV, CB) the diagonal above, so only a lane's edge
//     needs shuffles (two per step);
//   * row and column quantities are made once per pair, pass its lanes through a
//     ring in shared memory and move along the registers by one register (and
//     one byte permute) per two steps; the substitution costs are one table
//     lookup a cell;
//   * diagonals -40 and e0 (the band's boundary cells, which never carry a
//     finite value into the band but for row 0 and column 0) are infinite:
//     forced by the mask that clears the rank bits.  Row 0 is written by a
//     second copy of the step that runs while row 0 is inside the band (t <= e0);
//     column 0 follows from the ordinary rule.  Cells outside the matrix have
//     zero costs, so infinity stays infinity.
// Ranks.  Values are x4 when directions are wanted, the two low bits free: a
// minimum takes its candidates tagged with the rank of the reference's tie
// rule, as in k_aff_dp2.  The code byte of a cell is the sum of (tagged -
// cleared) times its weight, all multiply-adds: bits 0-1 todo, bit 2 the
// vertical move extends (END_VERTICAL's complement), bit 3 horizontal, bit 4
// diagonal, bits 5-6 the align choice.
//
// GAPS: some sequence has gap-bearing codes past position 0; without them the
// block-diagonal state is infinite everywhere and the openings are constant.
//
// Bound: integer issue (the ALU pipe 80 % busy).  Measured: 16,384 pairs of
// 100-5,000 bp with directions 27.4 ms in k_aff_dp2 and 3.2 ms here, their
// traceback 6.3 ms with a thread per pair and 0.7 ms with k_aff_walk; the costs
// of 38,001 pairs of 1,000 bp with gap-bearing codes 6.5 and 2.2 ms.
#include <algorithm>
#include <atomic>
#include "affine_diag.cuh"

namespace poyd {
namespace {

constexpr unsigned kDFull = 0xffffffffu;
constexpr unsigned kDInf2 = 0xC000C000u;
constexpr unsigned kDOne = 0x00010001u, kDTwo = 0x00020002u, kDRk = 0x00030003u;
constexpr unsigned kDClr = 0xFFFCFFFCu;
constexpr int kDWarps = 4;
constexpr int kDPad = 16;       // table row / column of a character outside the matrix
constexpr int kDStride = 18;    // entries per table row

struct DiagSmem {
  uint16_t sub[17 * kDStride];  // sc * cost[a & 15][b & 15]
  uint16_t rext[33], cext[33];  // sc * cost[a][gap], sc * cost[gap][b]
  uint16_t pad[12];
};
static_assert(sizeof(DiagSmem) % 16 == 0, "the rings after it are 16-byte aligned");

// Row and column quantities on their way to the registers, made once per pair
// and read by each of its lanes in turn: a ring per lane group and axis.  A
// chunk of C = D / 2 double steps brings C new ones; lane k reads C k places
// behind the first, so C times the lanes are alive (at most 8 a lane).
constexpr int kDRing = 8 * 32;  // records of a warp and axis, over its groups
template <bool GAPS>
struct DiagRec;
template <>
struct DiagRec<true> {  // x: v | o << 16, y: s | g << 16, z: table offset
  uint4 w;
};
template <>
struct DiagRec<false> {  // x: v, y: table offset
  uint2 w;
};
template <bool GAPS>
constexpr uint32_t diag_smem() {
  return sizeof(DiagSmem) + kDWarps * 2 * kDRing * sizeof(DiagRec<GAPS>);
}

__device__ __forceinline__ unsigned d_prmt(unsigned a, unsigned b, unsigned s) {
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}
__device__ __forceinline__ unsigned d_mad(unsigned a, unsigned b, unsigned c) {
  unsigned d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ unsigned d_sel(unsigned a, unsigned b, unsigned m) {  // b where m
  return (a & ~m) | (b & m);
}

template <bool GAPS, int D>
struct DiagState {
  static constexpr int NQ = D / 4, C = D / 2;
  // states of the two parities: x 0 even, 1 odd
  unsigned eh[2][NQ], ev[2][NQ], cb[2][NQ], eb[2][GAPS ? NQ : 1];
  // rows: vertical extension, opening + extension, opening, gap bit
  unsigned rv[NQ], ro[GAPS ? NQ : 1], rs[GAPS ? NQ : 1], rg[GAPS ? NQ : 1];
  // columns likewise
  unsigned cv[NQ], co[GAPS ? NQ : 1], cs[GAPS ? NQ : 1], cg[GAPS ? NQ : 1];
  unsigned keep[2][NQ], inf[2][NQ];  // masks of the band
  unsigned arow[C], bcol[C + 1];     // byte offsets of the cells' table rows / columns
  unsigned acc[2][NQ];               // code bytes of two double steps
};

// The step of parity X (0 even, 1 odd).  START: row 0 may be inside the band.
template <bool BT, bool GAPS, int D, int X, bool START>
__device__ __forceinline__ void diag_step(DiagState<GAPS, D> &S, const DiagSmem &sm, int src,
                                          unsigned go2, int i0, bool origin, bool odd,
                                          const AffDiagArgs &A) {
  constexpr int NQ = D / 4, Y = 1 - X;
  // the other parity's edge registers: d - 1 of the lane's first even cell is
  // the lane below's last odd one, d + 1 of its last odd cell the lane above's
  // first even one (a ring: the first and last indices are outside the band)
  unsigned edge1, edge2;  // EH or EV, CB of the neighbour
  if (X == 0) {
    edge1 = d_prmt(__shfl_sync(kDFull, S.eh[Y][NQ - 1], src), S.eh[Y][NQ - 1], 0x5432);
    edge2 = d_prmt(__shfl_sync(kDFull, S.cb[Y][NQ - 1], src), S.cb[Y][NQ - 1], 0x5432);
  } else {
    edge1 = d_prmt(S.ev[Y][0], __shfl_sync(kDFull, S.ev[Y][0], src), 0x5432);
    edge2 = d_prmt(S.cb[Y][0], __shfl_sync(kDFull, S.cb[Y][0], src), 0x5432);
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    // left (d - 1) and upper (d + 1) predecessors
    const unsigned ehl = X == 0 ? (q ? S.eh[Y][q ? q - 1 : 0] : edge1) : S.eh[Y][q];
    const unsigned cbl = X == 0 ? (q ? S.cb[Y][q ? q - 1 : 0] : edge2) : S.cb[Y][q];
    const unsigned evu = X == 0 ? S.ev[Y][q] : (q + 1 < NQ ? S.ev[Y][q + 1 < NQ ? q + 1 : 0] : edge1);
    const unsigned cbu = X == 0 ? S.cb[Y][q] : (q + 1 < NQ ? S.cb[Y][q + 1 < NQ ? q + 1 : 0] : edge2);
    const unsigned ehd = S.eh[X][q], evd = S.ev[X][q], cbd = S.cb[X][q];
    // substitution costs of the two cells
    const unsigned char *t = reinterpret_cast<const unsigned char *>(sm.sub);
    const unsigned lo =
        *reinterpret_cast<const uint16_t *>(t + d_mad(S.arow[q], A.one, S.bcol[q + X]));
    const unsigned hi =
        *reinterpret_cast<const uint16_t *>(t + d_mad(S.arow[q + NQ], A.one, S.bcol[q + NQ + X]));
    const unsigned cd = d_mad(hi, 65536u, lo);
    // FILL_EXTEND_HORIZONTAL / _VERTICAL: the opening (rank 0) wins ties
    // against the extension (rank 1)
    unsigned ehr, evr;
    if (GAPS) {
      ehr = __viaddmin_u16x2(ehl, BT ? S.cv[q] | kDOne : S.cv[q], d_mad(cbl, A.one, S.co[q]));
      evr = __viaddmin_u16x2(evu, BT ? S.rv[q] | kDOne : S.rv[q], d_mad(cbu, A.one, S.ro[q]));
    } else {
      ehr = d_mad(__viaddmin_u16x2(cbl, go2, BT ? d_mad(ehl, A.one, kDOne) : ehl), A.one, S.cv[q]);
      evr = d_mad(__viaddmin_u16x2(cbu, go2, BT ? d_mad(evu, A.one, kDOne) : evu), A.one, S.rv[q]);
    }
    // FILL_CLOSE_BLOCK_DIAGONAL: ranks horizontal 0, diagonal 1, vertical 2,
    // align 3; FILL_EXTEND_BLOCK_DIAGONAL[_NOBT]
    unsigned cbr, ebr = 0, eb = kDInf2;
    if (GAPS) {
      const unsigned ebd = S.eb[X][q];
      const unsigned both = S.rg[q] & S.cg[q];
      unsigned a = BT ? d_mad(cbd, A.one, kDRk) : cbd;
      a = __viaddmin_u16x2(evd, (S.cs[q] & S.rg[q]) | (BT ? kDTwo : 0u), a);
      a = __viaddmin_u16x2(ehd, S.rs[q] & S.cg[q], a);
      a = __viaddmin_u16x2(ebd, S.cs[q] | S.rs[q] | (BT ? kDOne : 0u), a);
      cbr = d_mad(a, A.one, cd);
      ebr = BT ? __viaddmin_u16x2(ebd, kDOne, cbd) : __vminu2(ebd, d_mad(go2, 2u, cbd));
      eb = d_sel(kDInf2, BT ? ebr & kDClr : ebr, both);
    } else {
      unsigned a = BT ? d_mad(cbd, A.one, kDRk) : cbd;
      a = BT ? __viaddmin_u16x2(evd, kDTwo, a) : __vminu2(evd, a);
      a = __vminu2(ehd, a);
      cbr = d_mad(a, A.one, cd);
    }
    // clear the ranks and force the cells outside the band.  The codes need
    // the cleared values before the forcing where a forced low half shares the
    // register with a cell of the band (index 0, in E[0]).
    // (Without ranks EH needs it at index 0 alone: above the band only EV and
    // CB are read by a cell of the band.)
    unsigned eh = BT || (X == 0 && q == 0) ? (ehr & S.keep[X][q]) | S.inf[X][q] : ehr;
    unsigned ev = (evr & S.keep[X][q]) | S.inf[X][q], cb = (cbr & S.keep[X][q]) | S.inf[X][q];
    if (BT) {
      const bool split = X == 0 && q == 0;
      const unsigned yh = split ? ehr & kDClr : eh, yv = split ? evr & kDClr : ev,
                     yc = split ? cbr & kDClr : cb;
      // ASSIGN_MINIMUM's choice: ranks EH 0, CB 1, EV 2, EB 3
      unsigned f = __viaddmin_u16x2(cb, kDOne, eh);
      f = __viaddmin_u16x2(ev, kDTwo, f);
      if (GAPS) f = __viaddmin_u16x2(eb, kDRk, f);
      unsigned code = d_mad(evr, A.k4, f & kDRk);
      code = d_mad(ehr, A.k8, code);
      code = d_mad(cbr, A.k32, code);
      unsigned clr = d_mad(yh, A.k8 >> 2, yv);        // (4 yv + 8 yh + 32 yc) / 4
      clr = d_mad(yc, A.k32 >> 2, clr);
      if (GAPS) {
        // eb is not infinite where its code is read
        code = d_mad(ebr, A.k16, code);
        clr = d_mad(ebr & kDClr, A.k4, clr);
      }
      code = d_mad(clr, A.m1 * 4u, code);
      S.acc[X][q] = odd ? d_mad(code, A.k256, S.acc[X][q]) : code;
    }
    if (START) {
      // row 0 (initialize_matrices_affine): cell c = i0 of the lane
      const unsigned m0 = (i0 == q ? 0xFFFFu : 0u) | (i0 == q + NQ ? 0xFFFF0000u : 0u);
      if (m0) {
        // EH extends without an opening; CB equals it; EV and EB infinite
        unsigned e = GAPS ? ehl + S.co[q] - S.cs[q] : ehl + S.cv[q];
        unsigned c = e, v = kDInf2, b = kDInf2;
        if (origin) e = v = go2, c = b = 0u;
        eh = d_sel(eh, e, m0);
        cb = d_sel(cb, c, m0);
        ev = d_sel(ev, v, m0);
        eb = d_sel(eb, b, m0);
      }
    }
    S.eh[X][q] = eh;
    S.ev[X][q] = ev;
    S.cb[X][q] = cb;
    if (GAPS) S.eb[X][q] = eb;
  }
}

// A row enters at the registers' first cell, a column at their last.  HI: the
// quantity is the high half of x.
template <int NQ, bool HI>
__device__ __forceinline__ void diag_shift_row(unsigned (&w)[NQ], unsigned x) {
  const unsigned last = w[NQ - 1];
#pragma unroll
  for (int q = NQ - 1; q > 0; --q) w[q] = w[q - 1];
  w[0] = d_prmt(x, last, HI ? 0x5432 : 0x5410);
}
template <int NQ, bool HI>
__device__ __forceinline__ void diag_shift_col(unsigned (&w)[NQ], unsigned x) {
  const unsigned first = w[0];
#pragma unroll
  for (int q = 0; q + 1 < NQ; ++q) w[q] = w[q + 1];
  w[NQ - 1] = d_prmt(first, x, HI ? 0x7632 : 0x5432);
}
template <bool GAPS, int D>
__device__ __forceinline__ void diag_row(DiagState<GAPS, D> &S, const DiagRec<GAPS> &r) {
  constexpr int NQ = D / 4;
  unsigned tab;
  diag_shift_row<NQ, false>(S.rv, r.w.x);
  if constexpr (GAPS) {
    diag_shift_row<NQ, true>(S.ro, r.w.x);
    diag_shift_row<NQ, false>(S.rs, r.w.y);
    diag_shift_row<NQ, true>(S.rg, r.w.y);
    tab = r.w.z;
  } else {
    tab = r.w.y;
  }
#pragma unroll
  for (int c = D / 2 - 1; c > 0; --c) S.arow[c] = S.arow[c - 1];
  S.arow[0] = tab;
}
template <bool GAPS, int D>
__device__ __forceinline__ void diag_col(DiagState<GAPS, D> &S, const DiagRec<GAPS> &r) {
  constexpr int NQ = D / 4;
  diag_shift_col<NQ, false>(S.cv, r.w.x);
  if constexpr (GAPS) {
    diag_shift_col<NQ, true>(S.co, r.w.x);
    diag_shift_col<NQ, false>(S.cs, r.w.y);
    diag_shift_col<NQ, true>(S.cg, r.w.y);
  }
}
template <bool GAPS, int D>
__device__ __forceinline__ void diag_col_char(DiagState<GAPS, D> &S, const DiagRec<GAPS> &r) {
#pragma unroll
  for (int x = 0; x < D / 2; ++x) S.bcol[x] = S.bcol[x + 1];
  if constexpr (GAPS) S.bcol[D / 2] = r.w.z;
  else S.bcol[D / 2] = r.w.y;
}

// A lane's pair and its places in it: its first cell's row and column are i0 +
// m and j0 + m at double step m; its group's rings.
template <bool GAPS>
struct DiagLane {
  const uint8_t *si, *sj;
  int leni, lenj, i0, j0;
  unsigned go, go2;
  DiagRec<GAPS> *rows, *cols;
  int mask;         // places of a ring - 1
  int below, above; // the group's lanes before and after this one, in a ring
  int c[4];  // characters of the next chunk's record: row, row before, column, before
};

__device__ __forceinline__ int diag_at(const uint8_t *s, int x, int len) {
  return x >= 0 && x <= len ? (int)__ldg(s + x) : 0;
}

// Quantities of row or column x (character c, the one before p), 0 outside the
// matrix: extension, opening + extension, opening, gap bit; table offset.
template <bool GAPS>
__device__ __forceinline__ DiagRec<GAPS> diag_rec(int x, int len, int c, int p, const uint16_t *ext,
                                                  unsigned go, unsigned stride) {
  const bool in = x >= 0 && x <= len;
  const unsigned e = in ? ext[c] : 0u;
  const unsigned tab = (in && x > 0 ? (unsigned)(c & 15) : (unsigned)kDPad) * stride;
  DiagRec<GAPS> r;
  if constexpr (GAPS) {
    const bool cg = (c & 16) != 0, pg = (p & 16) != 0;
    const unsigned s = !in || (!pg && cg) ? 0u : go;
    const unsigned v = x > 1 && pg && !cg ? s + e : e;
    r.w = make_uint4(v | (s + e) << 16, s | (in && cg ? 0xFFFF0000u : 0u), tab, 0u);
  } else {
    r.w = make_uint2(e, tab);
  }
  return r;
}

// The chunk of C rows from row and C columns from col into the rings (a lane a
// place); the characters were loaded a chunk before.
template <bool GAPS, int D>
__device__ __forceinline__ void diag_chars(DiagLane<GAPS> &L, int k, int row, int col) {
  L.c[0] = diag_at(L.si, row + k, L.leni);
  L.c[1] = diag_at(L.si, row + k - 1, L.leni);
  L.c[2] = diag_at(L.sj, col + k, L.lenj);
  L.c[3] = diag_at(L.sj, col + k - 1, L.lenj);
}
template <bool GAPS, int D>
__device__ __forceinline__ void diag_produce(DiagLane<GAPS> &L, const DiagSmem &sm, int k, int row,
                                             int col) {
  constexpr int C = D / 2;
  static_assert(C <= 8, "a lane a place");
  __syncwarp();  // the places written over have been read
  if (k < C) {
    L.rows[(row + k) & L.mask] =
        diag_rec<GAPS>(row + k, L.leni, L.c[0], L.c[1], sm.rext, L.go, 2 * kDStride);
    L.cols[(col + k) & L.mask] = diag_rec<GAPS>(col + k, L.lenj, L.c[2], L.c[3], sm.cext, L.go, 2);
  }
  diag_chars<GAPS, D>(L, k, row + C, col + C);
  __syncwarp();
}

// The least state of the cells of register q, parity x.
template <bool GAPS, int D>
__device__ __forceinline__ unsigned diag_least(const DiagState<GAPS, D> &S, int x, int fq) {
  unsigned w = 0;
#pragma unroll
  for (int q = 0; q < D / 4; ++q) {
    unsigned y = __vminu2(__vminu2(S.eh[x][q], S.ev[x][q]), S.cb[x][q]);
    if (GAPS) y = __vminu2(y, S.eb[x][q]);
    w = q == fq ? y : w;
  }
  return w;
}

// Double step m: row i0 + m and column j0 + C + m enter (bcol[c] is then column
// j0 + m + c; the odd step's last cell reads the new one).  CHECK: some pair's
// final cell or the task's last step may be this one.
template <bool BT, bool GAPS, int D, bool START, bool CHECK>
__device__ __forceinline__ void diag_double(DiagState<GAPS, D> &S, const DiagLane<GAPS> &L,
                                            const DiagSmem &sm, int m, bool odd, int last, int fin,
                                             int fq, unsigned &res, uint2 *dw,
                                            const AffDiagArgs &A) {
  constexpr int NQ = D / 4, C = D / 2;
  diag_row<GAPS, D>(S, L.rows[(L.i0 + m) & L.mask]);
  const DiagRec<GAPS> r = L.cols[(L.j0 + C + m) & L.mask];
  diag_col_char<GAPS, D>(S, r);
  diag_step<BT, GAPS, D, 0, START>(S, sm, L.below, L.go2, L.i0 + m, m == 0, odd, A);
  if (CHECK && 2 * m == fin) res = diag_least<GAPS, D>(S, 0, fq);
  diag_col<GAPS, D>(S, r);
  diag_step<BT, GAPS, D, 1, START>(S, sm, L.above, L.go2, L.i0 + m, false, odd, A);
  if (CHECK && 2 * m + 1 == fin) res = diag_least<GAPS, D>(S, 1, fq);
  if (BT && (odd || (CHECK && m == last))) {
    unsigned w[C];
#pragma unroll
    for (int q = 0; q < NQ; ++q) w[q] = S.acc[0][q], w[NQ + q] = S.acc[1][q];
#pragma unroll
    for (int v = 0; v < NQ; ++v)
      dw[((int64_t)(m >> 1) * NQ + v) * 32] = make_uint2(w[2 * v], w[2 * v + 1]);
  }
}

template <bool BT, bool GAPS, int D>
__device__ __forceinline__ void diag_task(const AffDiagArgs &A, const DiagSmem &sm,
                                          uint8_t *rings, int task, int64_t off, int lanes,
                                          int lane) {
  constexpr int NQ = D / 4, C = D / 2;
  constexpr int sc = BT ? 4 : 1;
  const int grp = lane / lanes, k = lane & (lanes - 1);
  const int id = A.order[task * kDiagTask + grp];
  DiagLane<GAPS> L;
  L.si = L.sj = A.seq;
  L.leni = L.lenj = -1;
  int e0 = 0;
  bool has = false;
  if (id >= 0) {
    const AffPlan P = A.plans[id];
    if (P.empty) {
      if (k == 0) A.cost[id] = 0;
    } else {
      has = true;
      L.leni = P.leni, L.lenj = P.lenj, e0 = P.e0;
      L.si += P.si_off, L.sj += P.sj_off;
    }
  }
  if (BT && has && k == 0) A.where[id] = AffWhere{off, lane, D};
  const int fin = has ? L.leni + L.lenj : -1;  // the final cell's step
  const int last = __reduce_max_sync(kDFull, fin >> 1), row0 = __reduce_max_sync(kDFull, e0) >> 1;
  const int fidx = L.lenj - L.leni + 40, fk = fidx / D, fc = fidx % D >> 1;  // its index
  L.go = (unsigned)(sc * A.go);
  L.go2 = L.go * 0x10001u;
  L.i0 = 20 - C * k;
  L.j0 = C * k - 20;

  DiagState<GAPS, D> S;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      S.eh[x][q] = S.ev[x][q] = S.cb[x][q] = kDInf2;
      if (GAPS) S.eb[x][q] = kDInf2;
      S.keep[x][q] = S.inf[x][q] = 0;
      S.acc[x][q] = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int idx = D * k + 2 * (q + h * NQ) + x;
        const bool in = idx > 0 && idx < e0 + 40;
        S.keep[x][q] |= (in ? (BT ? 0xFFFCu : 0xFFFFu) : 0u) << (16 * h);
        S.inf[x][q] |= (in ? 0u : 0xC000u) << (16 * h);
      }
    }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    S.rv[q] = S.cv[q] = 0;
    if (GAPS) S.ro[q] = S.rs[q] = S.rg[q] = S.co[q] = S.cs[q] = S.cg[q] = 0;
  }
#pragma unroll
  for (int c = 0; c < C; ++c) S.arow[c] = kDPad * 2 * kDStride;
#pragma unroll
  for (int c = 0; c <= C; ++c) S.bcol[c] = kDPad * 2;
  L.mask = 8 * lanes - 1;
  L.rows = reinterpret_cast<DiagRec<GAPS> *>(rings) + 2 * grp * 8 * lanes;
  L.cols = L.rows + 8 * lanes;
  L.below = (lane - k) | ((k - 1) & (lanes - 1));
  L.above = (lane - k) | ((k + 1) & (lanes - 1));
  // chunk of double steps m .. m + C - 1: rows 20 + m .. and columns col0 + m .. are
  // new (the first lane's rows and the last one's columns)
  const int col0 = lanes * C - 20;
#pragma unroll 1
  for (int m = -lanes * C; m <= -C; m += C) {
    diag_chars<GAPS, D>(L, k, 20 + m, col0 + m);
    diag_produce<GAPS, D>(L, sm, k, 20 + m, col0 + m);
  }
#pragma unroll 1
  for (int m = -C; m < 0; ++m) {  // the registers' first rows and columns
    diag_row<GAPS, D>(S, L.rows[(L.i0 + m) & L.mask]);
    const DiagRec<GAPS> r = L.cols[(L.j0 + C + m) & L.mask];
    diag_col_char<GAPS, D>(S, r);
    diag_col<GAPS, D>(S, r);
  }
  unsigned res = 0;
  uint2 *dw = BT ? reinterpret_cast<uint2 *>(A.dm + off) + lane : nullptr;
#pragma unroll 1
  for (int m = 0; m <= last; m += C) {
    diag_produce<GAPS, D>(L, sm, k, 20 + m, col0 + m);
    if (m <= row0) {
#pragma unroll 1
      for (int u = m; u < m + C && u <= last; ++u)
        diag_double<BT, GAPS, D, true, true>(S, L, sm, u, u & 1, last, fin, fc % NQ, res, dw, A);
    } else if (__any_sync(kDFull, fin >= 2 * m && fin < 2 * (m + C)) || m + C > last) {
#pragma unroll 1
      for (int u = m; u < m + C && u <= last; ++u)
        diag_double<BT, GAPS, D, false, true>(S, L, sm, u, u & 1, last, fin, fc % NQ, res, dw, A);
    } else {
      // the registers rotate by one place per double step: C of them unrolled
      // bring them back (two turns of the packed ones), with no moves
#pragma unroll
      for (int u = 0; u < C; ++u)
        diag_double<BT, GAPS, D, false, false>(S, L, sm, m + u, u & 1, last, fin, fc % NQ, res, dw, A);
    }
  }
  res = __shfl_sync(kDFull, res, (lane - k) + (has ? fk : 0));
  if (has && k == 0) A.cost[id] = (int)(res >> (16 * (fc / NQ)) & 0xFFFFu) / sc;
}

// SPREAD: the classes of a small batch with directions (a kernel of its own: the
// code for 8 diagonals a lane costs the others 2 %).
template <bool BT, bool GAPS, bool SPREAD>
__global__ void __launch_bounds__(kDWarps * 32, GAPS ? 3 : 4) k_aff_diag(const __grid_constant__ AffDiagArgs A) {
  extern __shared__ __align__(16) uint8_t diag_sm[];
  DiagSmem &sm = *reinterpret_cast<DiagSmem *>(diag_sm);
  uint8_t *rings = diag_sm + sizeof(DiagSmem) + (threadIdx.x >> 5) * 2 * kDRing * sizeof(DiagRec<GAPS>);
  constexpr int sc = BT ? 4 : 1;
  for (int e = threadIdx.x; e < 17 * kDStride; e += blockDim.x) {
    const int a = e / kDStride, b = e % kDStride;
    sm.sub[e] = a < 16 && b < 16 ? (uint16_t)(sc * (A.tables->packed[(a << 5) | b] & 0xffffu)) : 0;
  }
  for (int e = threadIdx.x; e < 33; e += blockDim.x) {
    sm.rext[e] = e < 32 ? (uint16_t)(sc * (A.tables->packed[(e << 5) | 16] & 0xffffu)) : 0;
    sm.cext[e] = e < 32 ? (uint16_t)(sc * (A.tables->packed[e] >> 16)) : 0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(A.counter, 1);
    t = __shfl_sync(kDFull, t, 0);
    if (t >= A.tasks) break;
    const int64_t word = A.task[t];
    const int64_t off = word & 0xFFFFFFFFFFFFll;
    const int lanes = (int)(word >> 56), width = (int)(word >> 48) & 0xFF;
    if (SPREAD && width == 8) diag_task<BT, GAPS, 8>(A, sm, rings, t, off, lanes, lane);
    else if (width == 12) diag_task<BT, GAPS, 12>(A, sm, rings, t, off, lanes, lane);
    else diag_task<BT, GAPS, 16>(A, sm, rings, t, off, lanes, lane);
  }
}

// backtrace_affine (algn.c:1983-2097) of one pair by a warp.  In align mode lane
// l reads the code l columns up the diagonal; the run up to the first cell that
// leaves the mode is taken at once.  A gap's first column is taken alone, the others
// likewise along the row or column: with a memory latency a column the walk of
// 200,000 pairs of 5 and 40 elements took 1.08 ms, 0.23 now, and a thread a pair
// (the rows kernels' walk) 0.13.  The block-diagonal mode takes a column at a time.
__global__ void __launch_bounds__(128) k_aff_walk(const __grid_constant__ AffWalkArgs A) {
  __shared__ uint8_t med[256];
  for (int t = threadIdx.x; t < 256; t += blockDim.x)
    med[t] = A.tables->median[(t >> 4) << 5 | (t & 15)];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int p = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  if (p >= A.n) return;
  const int id = A.order[p];
  if (id < 0) return;  // a task's missing pair
  const AffPlan P = A.plans[id];
  const int li = P.leni + 1, lj = P.lenj + 1;
  const int la = P.swap ? lj : li, lb = P.swap ? li : lj;
  const int64_t cap = slot_cap(la, lb);
  uint8_t *oa = A.out + A.out_off[id];
  uint8_t *ob = oa + cap, *ow = ob + cap, *om = ow + cap;
  const uint8_t *si = A.seq + P.si_off, *sj = A.seq + P.sj_off;
  if (P.empty) {
    const bool a_empty = P.empty == 1;
    const uint8_t *src = (a_empty != (bool)P.swap) ? sj : si;
    const int len = a_empty ? lb : la;
    for (int t = lane; t < len; t += 32) om[cap - len + t] = src[t];
    if (lane == 0) {
      A.out_len[2 * id] = 0;
      A.out_len[2 * id + 1] = len;
    }
    return;
  }
  uint8_t *ri = P.swap ? ob : oa, *rj = P.swap ? oa : ob;
  const AffWhere W = A.where[id];
  const int D = W.width, NQ = D / 4;
  const unsigned inv = 0xFFFFFFFFu / (unsigned)D + 1;  // idx / D
  const uint32_t *dm = A.dm + W.off + 2 * W.lane0;
  int i = P.leni, j = P.lenj, nr = 0, nm = 0, mode = 0, last_m = -1;
  bool bad = false;
  // columns of lanes below cnt: row character x, column character y (16: none),
  // the median byte md and whether the gap-free median takes it, mw with gaps
  auto emit = [&](int cnt, int x, int y, int md, bool keep, int mw) {
    const bool w = lane < cnt;
    const unsigned kb = __ballot_sync(kDFull, w && keep);
    if (w) {
      const int64_t q = cap - 1 - (nr + lane);
      ri[q] = (uint8_t)x;
      rj[q] = (uint8_t)y;
      ow[q] = (uint8_t)mw;
      if (keep) om[cap - 1 - (nm + __popc(kb & ((1u << lane) - 1u)))] = (uint8_t)md;
    }
    if (kb) last_m = __shfl_sync(kDFull, md, 31 - __clz(kb));
    nr += cnt;
    nm += __popc(kb);
  };
  while (i != 0 && j != 0) {
    const int idx = j - i + 40;
    if (idx <= 0 || idx >= P.e0 + 40 || nr + 4 >= cap) {  // left the band: a bug
      bad = true;
      break;
    }
    if (mode == 1 || mode == 2) {  // a gap past its first column: lane l the l-th of the rest
      const bool row = mode == 1;
      const int gi = row ? i - lane : i, gj = row ? j : j - lane, x = gj - gi + 40;
      const bool on = gi > 0 && gj > 0 && x > 0 && x < P.e0 + 40 && nr + lane + 4 < cap;
      unsigned go_on = 0;
      int ch = 16;
      if (on) {
        const int k = (int)__umulhi((unsigned)x, inv), c = (x - k * D) >> 1, m = (gi + gj) >> 1;
        const int w = ((x & 1) ? NQ : 0) + (c < NQ ? c : c - NQ);
        const uint32_t v = __ldcg(dm + (((int64_t)(m >> 1) * NQ + (w >> 1)) * 32 + k) * 2 + (w & 1));
        go_on = v >> ((c < NQ ? 0 : 16) + 8 * (m & 1)) & (row ? 4u : 8u);
        ch = (int)__ldg(row ? si + gi : sj + gj);
      }
      const unsigned stop = __ballot_sync(kDFull, !go_on), onb = __ballot_sync(kDFull, on);
      const int f = stop ? __ffs(stop) - 1 : 32;
      const bool ends = f < 32 && (onb >> f & 1u);
      const int cnt = f + ends;  // at least the first lane's, which the checks above let in
      emit(cnt, row ? ch : 16, row ? 16 : ch, ch | 16, !(ch & 16), (ch & 16) ? 16 : ch | 16);
      if (row) i -= cnt;
      else j -= cnt;
      if (ends) mode = 0;
      continue;
    }
    const int k = (int)__umulhi((unsigned)idx, inv), c = (idx - k * D) >> 1;
    const int qq = c < NQ ? c : c - NQ, half = c < NQ ? 0 : 16;
    const int w = ((idx & 1) ? NQ : 0) + qq;
    // lane l: cell (i - l, j - l)
    const int ii = i - lane, jj = j - lane, m = ((i + j) >> 1) - lane;
    const bool in = ii > 0 && jj > 0 && nr + lane + 4 < cap;
    unsigned code = 0;
    if (in) {
      const uint32_t x = __ldcg(dm + (((int64_t)(m >> 1) * NQ + (w >> 1)) * 32 + k) * 2 + (w & 1));
      code = (x >> (half + 8 * (m & 1))) & 0xFFu;
    }
    const unsigned c0 = __shfl_sync(kDFull, code, 0);
    if (mode == 0) mode = (c0 & 3u) == 0 ? 2 : (c0 & 3u) == 1 ? 4 : (c0 & 3u) == 2 ? 1 : 3;
    const int ic = in ? (int)__ldg(si + ii) : 16, jc = in ? (int)__ldg(sj + jj) : 16;
    if (mode == 4) {
      const unsigned a = (code >> 5) & 3u;
      const unsigned stop = __ballot_sync(kDFull, !in || a != 3u);
      const int f = stop ? __ffs(stop) - 1 : 32;
      const unsigned inb = __ballot_sync(kDFull, in);
      const int cnt = f < 32 && (inb >> f & 1u) ? f + 1 : f;
      const unsigned af = __shfl_sync(kDFull, a, f & 31);
      const int md = med[(ic & 15) << 4 | (jc & 15)];
      emit(cnt, ic, jc, md, true, md);
      i -= cnt;
      j -= cnt;
      if (cnt > f) mode = af == 0 ? 2 : af == 1 ? 3 : 1;
      continue;
    }
    if (mode == 1) {
      if (!(c0 & 4u)) mode = 0;
      emit(1, ic, 16, ic | 16, !(ic & 16), (ic & 16) ? 16 : ic | 16);
      --i;
    } else if (mode == 2) {
      if (!(c0 & 8u)) mode = 0;
      emit(1, 16, jc, jc | 16, !(jc & 16), (jc & 16) ? 16 : jc | 16);
      --j;
    } else {
      if (!(c0 & 16u)) mode = 0;
      emit(1, ic, jc, 0, false, 16);
      --i;
      --j;
    }
  }
  if (!bad) {
    // the rest of one sequence against gaps
    for (; i > 0; i -= min(i, 32)) {
      const int x = i - lane > 0 ? (int)__ldg(si + i - lane) : 16;
      emit(min(i, 32), x, 16, x | 16, !(x & 16), (x & 16) ? 16 : x | 16);
    }
    for (; j > 0; j -= min(j, 32)) {
      const int y = j - lane > 0 ? (int)__ldg(sj + j - lane) : 16;
      emit(min(j, 32), 16, y, y | 16, !(y & 16), (y & 16) ? 16 : y | 16);
    }
    // the leading gap; an empty median has no position 0 in the reference and
    // is treated as not a gap
    emit(1, 16, 16, 16, nm == 0 || last_m != 16, 16);
  }
  if (lane == 0) {
    A.out_len[2 * id] = bad ? -1 : nr;
    A.out_len[2 * id + 1] = bad ? -1 : nm;
  }
}

template <bool BT, bool GAPS, bool SPREAD = false>
void diag_launch(const AffDiagArgs &A, cudaStream_t st) {
  static std::atomic<int> cache[64];  // resident blocks of the device
  constexpr uint32_t sm = diag_smem<GAPS>();
  int dev = 0;
  cudaGetDevice(&dev);
  int c = cache[dev & 63].load();
  if (!c) {
    int per = 0, sms = 0;
    cudaFuncSetAttribute(k_aff_diag<BT, GAPS, SPREAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_aff_diag<BT, GAPS, SPREAD>, kDWarps * 32, sm);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cache[dev & 63].store(c = std::max(per, 1) * std::max(sms, 1));
  }
  k_aff_diag<BT, GAPS, SPREAD><<<std::min((A.tasks + kDWarps - 1) / kDWarps, c), kDWarps * 32, sm, st>>>(A);
}

}  // namespace

int launch_aff_diag(const AffDiagArgs &A, bool bt, bool gaps, bool spread, cudaStream_t st) {
  if (spread && gaps) diag_launch<true, true, true>(A, st);
  else if (spread) diag_launch<true, false, true>(A, st);
  else if (bt && gaps) diag_launch<true, true>(A, st);
  else if (bt) diag_launch<true, false>(A, st);
  else if (gaps) diag_launch<false, true>(A, st);
  else diag_launch<false, false>(A, st);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "k_aff_diag") : POYD_OK;
}

int launch_aff_walk(const AffWalkArgs &A, cudaStream_t st) {
  k_aff_walk<<<(A.n + 3) / 4, 128, 0, st>>>(A);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "k_aff_walk") : POYD_OK;
}

}  // namespace poyd
