// Three-sequence alignment without gap openings (go = 0, the linear model).
//
// With go = 0 a column's cost does not depend on the column before it
// (alignmentCost, ukkCommon.c:345-391, charges an opening per change of
// state), so the 16 states of a cell share one optimum: the cell's least
// cost over its states, and the lowest-numbered state that has it.  Kept
// together in 16 bits (cost x 16 + state) the recurrence over the seven
// neighbours n_d (d: the sequences that advance) is
//     M = min over d of (M(n_d) without its state) + 16 cost_d + state_d,
// state_d being the lowest-numbered of the cheapest states that advance d.
// The least cost and the tie rules are those of the 16-state kernel (k_p3):
// the walk's "lowest-numbered previous state" is the previous cell's own
// state, so four bits per cell replace sixteen choices.
//
// Bound: integer issue (7 add-mins, the mismatch terms and the choice bits
// per two cells: about 8 instructions a cell); the choices are 0.5 bytes a
// cell, the strip boundaries about 1.  Measured: 1,216 triples of 100-300 bp
// in 9.0 ms (10.1 with at most four warps a triple) where k_p3 with all 16 x 16
// state pairs took 339 ms.
//
// Layout.  The axes are the sequences by length: A the shortest, C the
// longest.  A thread owns a 4 x 4 tile of (A, B) and marches along C; its
// registers hold two cells each: rows 0-1 of A in the low halves at column
// c, rows 2-3 in the high halves at column c - 1, so the halves of a step do
// not depend on each other and one __viaddmin_u16x2 serves both.  Tiles are
// numbered row after row (f = ta * TB + tb); a warp takes 32 consecutive
// ones (a strip), lane k one column behind lane k - 1, from which it gets
// its B-neighbours by three shuffles.  Cells outside the cube need no test:
// infinity plus any cost stays infinite, and nothing in the cube reads a
// cell past its end.
// The A-neighbours come from the strips before: every tile writes its last
// row per step to a ring of strips in global memory (L2), and a warp brings
// the next 8 steps' rows into shared memory with cp.async while it computes
// 8.  The block's warps work on consecutive strips kP3LinLag = 48 steps apart
// (31 lanes + 8 steps of prefetch + 8 between barriers, rounded up to 8);
// a __syncthreads every 8 steps orders them.
#include <algorithm>
#include "three_kernels.cuh"

namespace poyd {
namespace {

__constant__ P3States c_p3l = p3_states();

constexpr unsigned kLinInf2 = 0xC000C000u;
constexpr int kMinTB = 17;  // tiles per row: a row's tile is read 16 steps after it is written

// The lowest-numbered of the cheapest states that advance e (bits: the
// sequences): one extension for one or two advancing sequences, none for
// three, plus the mismatches.
__host__ __device__ constexpr int lin_state(int e) {
  const P3States S = p3_states();
  const bool one = (e & (e - 1)) == 0;
  for (int t = 0; t < kP3States; ++t)
    if (S.adv[t] == e && (!one || S.ins[t])) return t;
  return 0;
}

struct LinArgs3 {
  P3Args A;
  uint8_t *plane;
  int64_t plane_stride;
  uint8_t *dir;
  int64_t dir_stride;
};

__device__ __forceinline__ unsigned p3_prmt(unsigned a, unsigned b, unsigned s) {
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}
__device__ __forceinline__ void p3_cp8(uint32_t dst, const void *src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void p3_cp16(uint32_t dst, const void *src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}

// Lengths past 0, axes and schedule of one triple.
struct LinGeo {
  int ax[3];         // sequence of axis A, B, C
  int na, nb, nc;    // last index per axis
  int TB, F, U, R;   // tiles per row, tiles, strips, ring strips
  int NS, P, W;      // steps per strip (of 8), strip period of a warp, warps
};

__device__ __forceinline__ LinGeo lin_geo(int la, int lb, int lc, int W) {
  LinGeo g;
  // stable sort of the three lengths: A shortest, C longest
  const int l[3] = {la, lb, lc};
  int a = 0, c = 0;
#pragma unroll
  for (int q = 1; q < 3; ++q) {
    if (l[q] < l[a]) a = q;
    if (l[q] >= l[c]) c = q;
  }
  const int b = 3 - a - c;
  g.ax[0] = a, g.ax[1] = b, g.ax[2] = c;
  g.na = (a == 0 ? la : a == 1 ? lb : lc) - 1;
  g.nb = (b == 0 ? la : b == 1 ? lb : lc) - 1;
  g.nc = (c == 0 ? la : c == 1 ? lb : lc) - 1;
  g.TB = max((g.nb + 4) >> 2, kMinTB);
  g.F = ((g.na + 4) >> 2) * g.TB;
  g.U = (g.F + 31) >> 5;
  g.R = ((g.TB + 31) >> 5) + 2;
  g.NS = (g.nc + 33 + 7) & ~7;
  g.W = W;
  g.P = max(g.NS, kP3LinLag * W);
  return g;
}

// One strip's per-lane inputs.
struct LinTile {
  unsigned K3[2][4];          // C_3 + the mismatch of A and B characters
  unsigned E[4], F[4];        // per A row / B column, byte q: 0x80 unless its base is q
  unsigned lz;                // all ones when the tile has no B-neighbour
};
struct LinRun {
  unsigned V[2][4];           // the tile at the last step
  unsigned U[4], L[2], LU;    // A-neighbours, B-neighbours and their corner, last step
};

template <int kW>
__global__ void __launch_bounds__(32 * kW) k_p3_linear(const __grid_constant__ LinArgs3 B) {
  const P3Args &A = B.A;
  extern __shared__ __align__(16) uint8_t lin3_sm[];
  __shared__ int s_job;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kThr = 32 * kW;
  // [warp][parity][8 steps][32 lanes] boundary words, [warp][parity][8] corner
  // records, then the columns' character selectors
  uint2 *st_row = reinterpret_cast<uint2 *>(lin3_sm) + warp * 2 * 8 * 32;
  uint4 *st_cor = reinterpret_cast<uint4 *>(lin3_sm + kW * 2 * 8 * 32 * 8) + warp * 2 * 8;
  uint16_t *sel = reinterpret_cast<uint16_t *>(lin3_sm + kW * 2 * 8 * (32 * 8 + 16));
  const uint32_t st_row_a = (uint32_t)__cvta_generic_to_shared(st_row);
  const uint32_t st_cor_a = (uint32_t)__cvta_generic_to_shared(st_cor);
  uint8_t *const plane = B.plane + blockIdx.x * B.plane_stride;
  uint32_t *const dir = reinterpret_cast<uint32_t *>(B.dir + blockIdx.x * B.dir_stride);
  const unsigned mm2 = 16u * A.mm * 0x10001u;
  const unsigned ge2 = 16u * A.ge * 0x10001u;

  for (;;) {
    __syncthreads();
    if (tid == 0) s_job = atomicAdd(A.counter, 1);
    __syncthreads();
    if (s_job >= A.n) break;
    const int i = A.order[s_job];
    const int la = A.len[0][i], lb = A.len[1][i], lc = A.len[2][i];
    const LinGeo g = lin_geo(la, lb, lc, kW);
    const int cq = g.ax[2];
    const uint8_t *sq[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int s = g.ax[q];
      sq[q] = A.seq + (s == 0 ? A.off[0][i] : s == 1 ? A.off[1][i] : A.off[2][i]);
    }
    // selector of column c (entry 32 + c): the low half's bytes take byte
    // q(c) of a lane's low word, the high half's byte q(c - 1) of its high
    // one, sign replicated
    for (int x = tid; x < g.NS + 40; x += kThr) sel[x] = 0xCC88;
    __syncthreads();
    // a character's bits go into its own column's entry (low half) and the
    // next one's (high half): written by bytes
    uint8_t *selb = reinterpret_cast<uint8_t *>(sel);
    const bool go_on = p3_begin(A, i, true, tid, kThr, [&](int q, int x, int code) {
      if (q == cq) {
        const int k = __ffs(code) - 1;
        selb[2 * (32 + x)] = (uint8_t)(0x88 | k * 0x11);
        selb[2 * (33 + x) + 1] = (uint8_t)(0xCC | k * 0x11);
      }
    });
    if (!go_on) continue;

    // costs x 16 + state per advancing axes d (bits A, B, C)
    unsigned Cd[8];
#pragma unroll
    for (int d = 1; d < 8; ++d) {
      const int e = (d & 1) << g.ax[0] | (d >> 1 & 1) << g.ax[1] | (d >> 2 & 1) << g.ax[2];
      int st = 0;
#pragma unroll
      for (int v = 1; v < 8; ++v) st = v == e ? lin_state(v) : st;
      Cd[d] = (d == 7 ? 0u : ge2) + (unsigned)st * 0x10001u;
    }
    const unsigned K7 = Cd[7] - Cd[3];  // per half: added to a value that holds C_3

    const int64_t row_bytes = (int64_t)g.NS * 256;         // a strip's boundary rows
    uint8_t *const cor = plane + (int64_t)g.R * row_bytes;  // a strip's corner records
    const int total = (g.U - 1) / kW * g.P + (g.U - 1) % kW * kP3LinLag + g.NS;
    auto strip_at = [&](int T, int &s) -> int {  // the warp's strip at time T and its step
      const int t = T - kP3LinLag * warp;
      if (t < 0) return -1;
      const int rd = t / g.P;
      s = t - rd * g.P;
      const int u = rd * kW + warp;
      return s < g.NS && u < g.U ? u : -1;
    };
    // the next chunk's inputs into stage `par`: this lane's A-neighbour row
    // (the tile f - TB at this lane's column) and lane 0's B-neighbours
    auto prefetch = [&](int u, int s, int par) {
      if (u >= 0) {
        const int src = 32 * u + lane - g.TB;
        const int us = src >> 5, dk = (src & 31) - lane + 1;
        const uint8_t *p = plane + (int64_t)(src >= 0 ? us % g.R : 0) * row_bytes + (src & 31) * 8;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const int sp = s + v + dk;
          const bool ok = src >= 0 && sp >= 0 && sp < g.NS;
          p3_cp8(st_row_a + ((par * 8 + v) * 32 + lane) * 8, p + (ok ? (int64_t)sp * 256 : 0), ok);
        }
        if (lane < 8) {
          const int sp = s + lane + 31;
          const bool ok = u > 0 && sp < g.NS;
          p3_cp16(st_cor_a + (par * 8 + lane) * 16,
                  cor + ((int64_t)(ok ? (u - 1) % g.R : 0) * g.NS + (ok ? sp : 0)) * 16, ok);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };

    LinTile X;
    LinRun S;
    unsigned acc[2][4];
    int par = 0;
    {
      int s = 0;
      const int u = strip_at(0, s);
      prefetch(u, s, 0);
    }
    for (int T = 0; T < total; T += 8, par ^= 1) {
      // the warp's own copies of this chunk, then everyone's rows of the last
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      {
        int s = 0;
        const int u = strip_at(T + 8, s);
        prefetch(u, s, par ^ 1);
      }
      int s = 0;
      const int u = strip_at(T, s);
      if (u < 0) continue;
      if (s == 0) {
        const int f = 32 * u + lane, ta = f / g.TB, tb = f - ta * g.TB;
        int qa[4], qb[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int a = 4 * ta + r, b = 4 * tb + r;
          qa[r] = a >= 1 && a <= g.na ? p3_ix(p3_code(sq[0][a])) : 0;
          qb[r] = b >= 1 && b <= g.nb ? p3_ix(p3_code(sq[1][b])) : 0;
          X.E[r] = 0x80808080u ^ (0x80u << (8 * qa[r]));
          X.F[r] = 0x80808080u ^ (0x80u << (8 * qb[r]));
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const unsigned ne = (qa[r] != qb[q] ? 0xFFFFu : 0u) | (qa[r + 2] != qb[q] ? 0xFFFF0000u : 0u);
            X.K3[r][q] = Cd[3] + (ne & mm2);
            S.V[r][q] = kLinInf2;
          }
#pragma unroll
        for (int q = 0; q < 4; ++q) S.U[q] = kLinInf2;
        S.L[0] = S.L[1] = S.LU = kLinInf2;
        X.lz = tb == 0 ? ~0u : 0u;
      }
      uint2 *const row_out =
          reinterpret_cast<uint2 *>(plane + (int64_t)(u % g.R) * row_bytes) + lane;
      uint4 *const cor_out = reinterpret_cast<uint4 *>(cor) + (int64_t)(u % g.R) * g.NS;
      const uint2 *in_row = st_row + par * 8 * 32 + lane;
      const uint4 *in_cor = st_cor + par * 8;
      const uint16_t *selp = sel + 32 + s - lane;
      uint4 *const dw = reinterpret_cast<uint4 *>(dir) + ((int64_t)u * (g.NS / 4) + s / 4) * 64 + lane;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        // boundary words are stored xor infinity: a row outside the cube
        // (zero-filled) is infinite
        const uint2 rw = in_row[v * 32];
        const uint4 cw = in_cor[v];
        const unsigned sl = selp[v];
        unsigned r0 = __shfl_up_sync(0xffffffffu, S.V[0][3], 1);
        unsigned r1 = __shfl_up_sync(0xffffffffu, S.V[1][3], 1);
        unsigned r2 = __shfl_up_sync(0xffffffffu, S.U[3], 1);
        if (lane == 0) r0 = cw.x, r1 = cw.y, r2 = cw.z;
        const unsigned L0 = (r0 & ~X.lz) | (kLinInf2 & X.lz);
        const unsigned L1 = (r1 & ~X.lz) | (kLinInf2 & X.lz);
        const unsigned LU = (r2 & ~X.lz) | (kLinInf2 & X.lz);
        unsigned U[4];
        const unsigned p0 = rw.x ^ kLinInf2, p1 = rw.y ^ kLinInf2;
        U[0] = p3_prmt(p0, S.V[1][0], 0x5410);
        U[1] = p3_prmt(p0, S.V[1][1], 0x5432);
        U[2] = p3_prmt(p1, S.V[1][2], 0x5410);
        U[3] = p3_prmt(p1, S.V[1][3], 0x5432);
        // mismatches with this step's C characters
        const unsigned n5[2] = {p3_prmt(X.E[0], X.E[2], sl), p3_prmt(X.E[1], X.E[3], sl)};
        const unsigned x5[2] = {(n5[0] & mm2) + Cd[5], (n5[1] & mm2) + Cd[5]};
        unsigned n6[4], x6[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          n6[q] = p3_prmt(X.F[q], X.F[q], sl);
          x6[q] = (n6[q] & mm2) + Cd[6];
        }
        unsigned N[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const unsigned up = r ? N[0][q] : U[q], upp = r ? S.V[0][q] : S.U[q];
            const unsigned lf = q ? N[r][q - 1] : (r ? L1 : L0);
            const unsigned lfp = q ? S.V[r][q - 1] : S.L[r];
            const unsigned ul = r ? (q ? N[0][q - 1] : L0) : (q ? U[q - 1] : LU);
            const unsigned ulp = r ? (q ? S.V[0][q - 1] : S.L[0]) : (q ? S.U[q - 1] : S.LU);
            const unsigned x7 = (n5[r] & n6[q] & mm2) + X.K3[r][q] + K7;
            unsigned m = __viaddmin_u16x2(S.V[r][q], Cd[4], kLinInf2);
            m = __viaddmin_u16x2(upp, x5[r], m);
            m = __viaddmin_u16x2(lfp, x6[q], m);
            m = __viaddmin_u16x2(ulp, x7, m);
            m = __viaddmin_u16x2(ul, X.K3[r][q], m);
            m = __viaddmin_u16x2(up, Cd[1], m);
            m = __viaddmin_u16x2(lf, Cd[2], m);
            if (v == 0 && r == 0 && q == 0 && u == 0 && s == 0 && lane == 0)
              m &= 0xFFFF0000u;  // the start: MMM at cost 0
            N[r][q] = m & 0xFFF0FFF0u;
            acc[r][q] = ((v & 3) ? acc[r][q] * 16 : 0u) + (m - N[r][q]);
          }
        // this tile's last row (the high halves, column c - 1) for the strip
        // below; lane 31's B-neighbours for the next strip's lane 0
        row_out[(s + v) * 32] = make_uint2(p3_prmt(N[1][0], N[1][1], 0x7632) ^ kLinInf2,
                                           p3_prmt(N[1][2], N[1][3], 0x7632) ^ kLinInf2);
        if (lane == 31) cor_out[s + v] = make_uint4(N[0][3], N[1][3], U[3], 0);
        S.L[0] = L0, S.L[1] = L1, S.LU = LU;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          S.U[q] = U[q];
          S.V[0][q] = N[0][q];
          S.V[1][q] = N[1][q];
        }
        if ((v & 3) == 3) {
          dw[(v >> 2) * 64] = make_uint4(acc[0][0], acc[0][1], acc[0][2], acc[0][3]);
          dw[(v >> 2) * 64 + 32] = make_uint4(acc[1][0], acc[1][1], acc[1][2], acc[1][3]);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
      auto nib = [&](int x, int y, int z) -> int {
        const int a = g.ax[0] == 0 ? x : g.ax[0] == 1 ? y : z;
        const int b = g.ax[1] == 0 ? x : g.ax[1] == 1 ? y : z;
        const int c = g.ax[2] == 0 ? x : g.ax[2] == 1 ? y : z;
        const int f = (a >> 2) * g.TB + (b >> 2), k = f & 31, h = a >> 1 & 1, s = k + c + h;
        const int64_t w = ((int64_t)(f >> 5) * (g.NS / 4) + (s >> 2)) * 256 + (a & 1) * 128 + k * 4 + (b & 3);
        return (int)(__ldcg(dir + w) >> (16 * h + 4 * (3 - (s & 3)))) & 15;
      };
      // an optimum of 0xC000 / 16 or more reached the clamp: redo in 32 bits
      if (!p3_walk_states(A, c_p3l, i, lane, 0xC00, nib) && lane == 0) atomicOr(A.err, 4);
    }
  }
}

constexpr size_t lin3_smem(int warps, int longest) {
  return (size_t)warps * 2 * 8 * (32 * 8 + 16) + 2 * ((size_t)longest + 40 + 48);
}

template <int kW>
int lin3_blocks(int longest) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t sm = lin3_smem(kW, longest);
  // The same request for every batch: it is one value per kernel and device, which
  // a thread with shorter sequences would lower under another's launch.
  constexpr size_t most = lin3_smem(kW, kP3MaxLen);
  if (most > 48 * 1024)
    cudaFuncSetAttribute(k_p3_linear<kW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_p3_linear<kW>, 32 * kW, sm) != cudaSuccess)
    per = 1;
  return std::max(per, 1) * std::max(sms, 1);
}

}  // namespace

P3LinearPlan p3_linear_plan(int64_t la, int64_t lb, int64_t lc) {
  int64_t l[3] = {la, lb, lc};
  std::sort(l, l + 3);
  const int64_t TB = std::max<int64_t>((l[1] + 3) / 4, kMinTB), F = (l[0] + 3) / 4 * TB;
  const int64_t U = (F + 31) / 32, R = (TB + 31) / 32 + 2, NS = (l[2] + 32 + 7) & ~(int64_t)7;
  return {R * NS * (256 + 16), U * NS * 256};
}

int64_t p3_linear_steps(int64_t la, int64_t lb, int64_t lc) {
  const P3LinearPlan p = p3_linear_plan(la, lb, lc);
  return p.dir / 256;
}

int64_t p3_linear_chain(int64_t la, int64_t lb, int64_t lc, int warps) {
  const P3LinearPlan p = p3_linear_plan(la, lb, lc);
  const int64_t NS = (std::max({la, lb, lc}) + 32 + 7) & ~(int64_t)7, U = p.dir / 256 / NS;
  return (U - 1) / warps * std::max<int64_t>(NS, kP3LinLag * warps) + (U - 1) % warps * kP3LinLag + NS;
}

int p3_linear_blocks(int warps, int longest) {
  return warps == 1 ? lin3_blocks<1>(longest) : warps == 2 ? lin3_blocks<2>(longest)
       : warps == 4 ? lin3_blocks<4>(longest) : warps == 8 ? lin3_blocks<8>(longest)
                                              : lin3_blocks<16>(longest);
}

int launch_p3_linear(const P3Args &A, int warps, int longest, int blocks, uint8_t *plane,
                     int64_t plane_stride, uint8_t *dir, int64_t dir_stride, cudaStream_t st) {
  const LinArgs3 B = {A, plane, plane_stride, dir, dir_stride};
  const size_t sm = lin3_smem(warps, longest);
  ProfScope ps("p3", st);
  switch (warps) {
    case 1: k_p3_linear<1><<<blocks, 32, sm, st>>>(B); break;
    case 2: k_p3_linear<2><<<blocks, 64, sm, st>>>(B); break;
    case 4: k_p3_linear<4><<<blocks, 128, sm, st>>>(B); break;
    case 8: k_p3_linear<8><<<blocks, 256, sm, st>>>(B); break;
    default: k_p3_linear<16><<<blocks, 512, sm, st>>>(B); break;
  }
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "k_p3_linear") : POYD_OK;
}

}  // namespace poyd
