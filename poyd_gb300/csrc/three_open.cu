// Three-sequence alignment with gap openings (go > 0, the affine model), in
// 16-bit values.
//
// A cell holds the 16 column states' costs v[s] (x 16, the state's own number
// in the low bits, so that a minimum keeps the lowest-numbered state among
// equals).  What a later column in state t needs of a cell is
//     T[t] = min over s of v[s] + go * (openings of s -> t),
// and an opening is charged per sequence (ukkCommon.c:263-290: the sequence
// is in D or I in t and was not in that state in s), so the 16 x 16 minimum
// separates into three passes over the states of one sequence each: with m =
// min(M, D, I), M becomes m, D becomes min(D, m + go), I min(I, m + go).  75
// operations for all T instead of 256, made once at the cell instead of once
// per neighbour that reads it, and a neighbour then reads one value per state
// instead of 16: v'[t] = T[t] of the cell that t's column comes from, + col(t).
// Costs, choices and ties are those of the 32-bit kernel (k_p3), which takes
// batches whose values may not fit.
//
// Bound: integer issue (~130 instructions a cell, most on the half-rate ALU
// pipe), and for small batches the barriers.  Measured (20 triples of 150-200
// bp): 15 ms with 16 x 16 state pairs and a cluster barrier per hyperplane,
// 1.8 ms here with clusters of 6 blocks (8.9 ms with one block a triple, 2.3
// with clusters of 8, which do not all fit at once).
//
// Layout.  A warp takes two rows of sequence a by 32 of b (a task) and
// marches along c, lane k one column behind lane k - 1; a thread's registers
// hold {row a at column c, row a + 1 at column c - 1}, which do not depend on
// each other, so one __viaddmin_u16x2 serves both.  b-neighbours come by
// seven shuffles; a-neighbours from the task two rows up, through a ring in
// global memory (16 bytes per lane and step); the b-neighbour of lane 0 from
// the task to its left, through a 32-byte record per step.  Both are brought
// into shared memory 8 steps ahead with cp.async.  Tasks start kOpenLagA = 32
// steps after the one above (8 of prefetch, 16 until a chunk's stores are
// visible, one for the second row, rounded up to 8) and kOpenLagB = 56 after
// the one to the left (31 lanes more); a barrier every 8 steps orders them.
// The warps of a block, or of a cluster of blocks when the batch is small,
// take the tasks round robin; a b longer than the warps' strips runs in panels.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include "three_kernels.cuh"

namespace poyd {
namespace {

__constant__ P3States c_p3o = p3_states();

constexpr unsigned kOInf2 = 0xC000C000u;
constexpr unsigned kOClear = 0xFFF0FFF0u;
constexpr int kOpenWarps = 8;
constexpr int kOpenLagA = 32, kOpenLagB = 56, kOpenRing = 3;

struct OpenArgs {
  P3Args A;
  uint8_t *plane;  // per triple slot: boundary ring, then left records
  int64_t plane_stride;
  uint8_t *dir;
  int64_t dir_stride;
  unsigned one, sixteen, m1;  // multipliers the compiler does not know: 1, 16, -1
};

// The states of one advance d (bits: the sequences), in increasing order.
struct OpenTargets {
  int n[8], t[8][4];
};
__host__ __device__ constexpr OpenTargets open_targets() {
  constexpr P3States S = p3_states();
  OpenTargets R{};
  for (int t = 0; t < kP3States; ++t) R.t[S.adv[t]][R.n[S.adv[t]]++] = t;
  return R;
}

__device__ __forceinline__ unsigned o_prmt(unsigned a, unsigned b, unsigned s) {
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}
// An add kept on the multiply-add pipe: the ALU pipe is the busier one.
__device__ __forceinline__ unsigned o_mad(unsigned a, unsigned b, unsigned c) {
  unsigned d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ void o_cp16(uint32_t dst, const void *src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}

// One sequence's pass of T (stride 1, 3 or 9 in the 27 combinations of M, D,
// I); h: which combinations hold a value.
template <int ST>
__device__ __forceinline__ void o_pass(unsigned (&x)[27], bool (&h)[27], unsigned go2, unsigned one) {
#pragma unroll
  for (int e = 0; e < 27; ++e) {
    if (e / ST % 3 != 0) continue;
    const int M = e, D = e + ST, I = e + 2 * ST;
    if (!h[M] && !h[D] && !h[I]) continue;
    unsigned m = h[M] ? x[M] : h[D] ? x[D] : x[I];
    if (h[M] && h[D]) m = __vminu2(m, x[D]);
    if ((h[M] || h[D]) && h[I]) m = __vminu2(m, x[I]);
    x[D] = h[D] ? __viaddmin_u16x2(m, go2, x[D]) : o_mad(m, one, go2);
    x[I] = h[I] ? __viaddmin_u16x2(m, go2, x[I]) : o_mad(m, one, go2);
    x[M] = m;
    h[M] = h[D] = h[I] = true;
  }
}

// CL: a cluster of blocks per triple.  CLAMP: T is cut off at infinity
// before the column cost is added (large costs; otherwise the sum cannot
// leave 16 bits).
template <bool CL, bool CLAMP>
__global__ void __launch_bounds__(32 * kOpenWarps, 2) k_p3_open(const __grid_constant__ OpenArgs B) {
  namespace cg = cooperative_groups;
  constexpr P3States S = p3_states();
  constexpr OpenTargets R = open_targets();
  const P3Args &A = B.A;
  extern __shared__ __align__(16) uint8_t open_sm[];
  __shared__ int s_job;
  __shared__ unsigned s_end;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kThr = 32 * kOpenWarps;
  const int rank = CL ? (int)cg::this_cluster().block_rank() : 0;
  const int csz = CL ? (int)cg::this_cluster().num_blocks() : 1;
  const int64_t slot = blockIdx.x / csz;
  auto bar = [&]() {
    if (CL) cg::this_cluster().sync();
    else __syncthreads();
  };
  uint4 *st_row = reinterpret_cast<uint4 *>(open_sm) + warp * 2 * 8 * 32;
  uint4 *st_cor = reinterpret_cast<uint4 *>(open_sm + kOpenWarps * 2 * 8 * 32 * 16) + warp * 2 * 8 * 2;
  uint16_t *sel = reinterpret_cast<uint16_t *>(open_sm + kOpenWarps * 2 * 8 * (32 + 2) * 16);
  const uint32_t st_row_a = (uint32_t)__cvta_generic_to_shared(st_row);
  const uint32_t st_cor_a = (uint32_t)__cvta_generic_to_shared(st_cor);
  uint8_t *const plane = B.plane + slot * B.plane_stride;
  uint4 *const dir = reinterpret_cast<uint4 *>(B.dir + slot * B.dir_stride);
  const unsigned mm2 = 16u * A.mm * 0x10001u, ge2 = 16u * A.ge * 0x10001u;
  const unsigned go2 = 16u * A.go * 0x10001u;

  for (;;) {
    bar();
    if (rank == 0 && tid == 0) s_job = atomicAdd(A.counter, 1);
    bar();
    const int job = CL ? *cg::this_cluster().map_shared_rank(&s_job, 0) : s_job;
    if (CL) cg::this_cluster().sync();  // every block has read block 0's s_job
    if (job >= A.n) break;
    const int i = A.order[job];
    const int la = A.len[0][i], lb = A.len[1][i], lc = A.len[2][i];
    const int na = la - 1, nb = lb - 1, nc = lc - 1;
    const int NS = (nc + 33 + 7) & ~7;         // steps of a task
    const int NR = (la + 1) >> 1;              // row pairs
    const int NB = (lb + 31) >> 5;             // strips of b
    const int Wt = csz * kOpenWarps;
    const int NP = min(NB, Wt);                // strips of a panel
    const int Rw = min(Wt / NP, (NS + kOpenLagA - 1) / kOpenLagA);  // row pairs in flight
    const int P = max(NS, Rw * kOpenLagA);     // a warp's period
    const uint8_t *s0 = A.seq + A.off[0][i], *s1 = A.seq + A.off[1][i];
    for (int x = tid; x < NS + 40; x += kThr) sel[x] = 0xCC88;
    __syncthreads();
    // selector of column c (entry 32 + c): byte q(c) of a lane's first word
    // for the low half, byte q(c - 1) of its second for the high half, sign
    // replicated
    uint8_t *selb = reinterpret_cast<uint8_t *>(sel);
    if (!p3_begin(A, i, rank == 0, tid, kThr, [&](int q, int x, int code) {
          if (q == 2) {
            const int k = __ffs(code) - 1;
            selb[2 * (32 + x)] = (uint8_t)(0x88 | k * 0x11);
            selb[2 * (33 + x) + 1] = (uint8_t)(0xCC | k * 0x11);
          }
        }))
      continue;

    const int64_t row_bytes = (int64_t)NS * 512;              // a task's boundary rows
    uint8_t *const left = plane + (int64_t)kOpenRing * NP * row_bytes;  // [row pair][strip][step] 32 B
    const int gid = rank * kOpenWarps + warp, vin = gid % NP, rin = gid / NP;
    const int dur = (NR - 1) / Rw * P + (NR - 1) % Rw * kOpenLagA + (NP - 1) * kOpenLagB + NS;
    // the task of the end cell and the step at which its lane meets it
    const int e_ra = na >> 1, e_v = nb >> 5, e_s = (nb & 31) + nc + (na & 1);
    unsigned Tp[kP3States];                       // T at the last step
    unsigned U3 = kOInf2, U5 = kOInf2, U7 = kOInf2, L6 = kOInf2, L7 = kOInf2;
    unsigned Er0 = 0, Er1 = 0, Fb = 0, n01 = 0, endv = 0;

    for (int v0 = 0; v0 < NB; v0 += NP) {
      const int v = v0 + vin;
      const bool mine = rin < Rw && v < NB;
      auto task_at = [&](int T, int &s) -> int {  // the warp's row pair at time T and its step
        const int t = T - rin * kOpenLagA - vin * kOpenLagB;
        if (t < 0 || !mine) return -1;
        const int rd = t / P;
        s = t - rd * P;
        const int ra = rd * Rw + rin;
        return s < NS && ra < NR ? ra : -1;
      };
      auto prefetch = [&](int ra, int s, int par) {
        if (ra >= 0) {
          const uint8_t *p =
              plane + ((int64_t)((ra + kOpenRing - 1) % kOpenRing) * NP + vin) * row_bytes + lane * 16;
#pragma unroll
          for (int u = 0; u < 8; ++u) {  // the row above at this lane's column: one step later there
            const bool ok = s + u + 1 < NS;  // else past its last column
            if (ra > 0)
              o_cp16(st_row_a + ((par * 8 + u) * 32 + lane) * 16, p + (ok ? (int64_t)(s + u + 1) * 512 : 0), ok);
            else
              st_row[(par * 8 + u) * 32 + lane] = make_uint4(kOInf2, kOInf2, kOInf2, kOInf2);
          }
          if (v > 0 && lane < 16) {
            const int sp = s + (lane >> 1) + 31;
            const bool ok = sp < NS;
            o_cp16(st_cor_a + (par * 16 + lane) * 16,
                   left + (((int64_t)ra * NB + v - 1) * NS + (ok ? sp : 0)) * 32 + (lane & 1) * 16, ok);
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      if (v0) bar();  // the last panel's records
      if (v == 0) {   // no b-neighbour
        st_cor[lane] = make_uint4(kOInf2, kOInf2, kOInf2, kOInf2);
        __syncwarp();
      }
      int par = 0;
      {
        int s = 0;
        const int ra = task_at(0, s);
        prefetch(ra, s, 0);
      }
      for (int T = 0; T < dur; T += 8, par ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // a cluster's barrier is in two halves, a chunk apart: what chunk
        // q - 2 wrote is visible in chunk q, and nobody waits for the stores
        // of the chunk just done
        if (CL) {
          __syncwarp();
          if (T) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
          asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        } else {
          __syncthreads();
        }
        {
          int s = 0;
          const int ra = task_at(T + 8, s);
          prefetch(ra, s, par ^ 1);
        }
        int s = 0;
        const int ra = task_at(T, s);
        if (ra < 0) continue;
        if (s == 0) {
          const int b = 32 * v + lane;
          const int q0 = 2 * ra >= 1 && 2 * ra <= na ? p3_ix(p3_code(s0[2 * ra])) : 0;
          const int q1 = 2 * ra + 1 <= na ? p3_ix(p3_code(s0[2 * ra + 1])) : 0;
          const int qb = b >= 1 && b <= nb ? p3_ix(p3_code(s1[b])) : 0;
          Er0 = 0x80808080u ^ (0x80u << (8 * q0));
          Er1 = 0x80808080u ^ (0x80u << (8 * q1));
          Fb = 0x80808080u ^ (0x80u << (8 * qb));
          n01 = ((q0 != qb ? 0xFFFFu : 0u) | (q1 != qb ? 0xFFFF0000u : 0u)) & mm2;
#pragma unroll
          for (int t = 0; t < kP3States; ++t) Tp[t] = kOInf2;
          U3 = U5 = U7 = L6 = L7 = kOInf2;
        }
        uint4 *const row_out =
            reinterpret_cast<uint4 *>(plane + ((int64_t)(ra % kOpenRing) * NP + vin) * row_bytes) + lane;
        uint4 *const left_out = reinterpret_cast<uint4 *>(left) + ((int64_t)ra * NB + v) * NS * 2;
        uint4 *const dw = dir + (((int64_t)ra * NB + v) * NS + s) * 32 + lane;
        const uint4 *in_row = st_row + par * 8 * 32 + lane;
        const uint4 *in_cor = st_cor + par * 16;
        const uint16_t *selp = sel + 32 + s - lane;
        const bool start = ra == 0 && v == 0 && s == 0 && lane == 0;
        const int cap = ra == e_ra && v == e_v && lane == (nb & 31) ? e_s - s : -1;
#pragma unroll 4
        for (int u = 0; u < 8; ++u) {
          const uint4 rw = in_row[u * 32];
          const uint4 c0 = in_cor[2 * u], c1 = in_cor[2 * u + 1];
          const unsigned sl = selp[u];
          unsigned X[kP3States];  // T of the cell each state comes from
          // c alone: this cell one column back
#pragma unroll
          for (int q = 0; q < 4; ++q) X[R.t[4][q]] = Tp[R.t[4][q]];
          // b, b + c, a + b, a + b + c: lane k - 1
          unsigned y[7];
#pragma unroll
          for (int q = 0; q < 4; ++q) y[q] = __shfl_up_sync(0xffffffffu, Tp[R.t[2][q]], 1);
          y[4] = __shfl_up_sync(0xffffffffu, Tp[R.t[6][0]], 1);
          y[5] = __shfl_up_sync(0xffffffffu, U3, 1);
          y[6] = __shfl_up_sync(0xffffffffu, U7, 1);
          if (lane == 0) {
            y[0] = c0.x, y[1] = c0.y, y[2] = c0.z, y[3] = c0.w;
            y[4] = c1.x, y[5] = c1.y, y[6] = c1.z;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) X[R.t[2][q]] = y[q];
          X[R.t[6][0]] = L6;
          X[R.t[7][0]] = L7;
          X[R.t[3][0]] = y[5];
          L6 = y[4];
          L7 = y[6];
          // a, a + c: the row above (low half: the task above; high half: this
          // thread's first row one step ago)
          X[R.t[1][0]] = o_prmt(rw.x, Tp[R.t[1][0]], 0x5410);
          X[R.t[1][1]] = o_prmt(rw.x, Tp[R.t[1][1]], 0x5432);
          X[R.t[1][2]] = o_prmt(rw.y, Tp[R.t[1][2]], 0x5410);
          X[R.t[1][3]] = o_prmt(rw.y, Tp[R.t[1][3]], 0x5432);
          X[R.t[5][0]] = U5;
          U5 = o_prmt(rw.z, Tp[R.t[5][0]], 0x5410);
          U3 = o_prmt(rw.z, Tp[R.t[3][0]], 0x5432);
          U7 = o_prmt(rw.w, Tp[R.t[7][0]], 0x5432);
          // the choices, four states a word (a nibble per half and state)
          uint4 w;
          unsigned *wp = &w.x;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            // sum of 16^q (X - X cleared), all multiply-adds (the ALU pipe is
            // the busier one); the true sum fits, whatever wraps on the way
            unsigned z = X[4 * k + 3], c = X[4 * k + 3] & kOClear;
#pragma unroll
            for (int q = 2; q >= 0; --q) {
              z = o_mad(z, B.sixteen, X[4 * k + q]);
              c = o_mad(c, B.sixteen, X[4 * k + q] & kOClear);
            }
            wp[k] = o_mad(c, B.m1, z);
          }
          dw[u * 32] = w;
          // column costs: one extension per D, one for an I; mismatches of the
          // advancing sequences
          const unsigned n5 = o_prmt(Er0, Er1, sl), n6 = o_prmt(Fb, Fb, sl);
          unsigned x[27];
          bool h[27];
#pragma unroll
          for (int e = 0; e < 27; ++e) h[e] = false, x[e] = 0;
#pragma unroll
          for (int t = 0; t < kP3States; ++t) {
            const unsigned own = (unsigned)t * 0x10001u;
            unsigned col = S.ins[t] ? ge2 : S.ndel[t] == 2 ? 2 * ge2 : S.ndel[t] == 1 ? ge2 : 0u;
            if (S.adv[t] == 3) col = o_mad(n01, B.one, col);
            if (S.adv[t] == 5) col = o_mad(n5 & mm2, B.one, col);
            if (S.adv[t] == 6) col = o_mad(n6 & mm2, B.one, col);
            if (S.adv[t] == 7) col = o_mad(n01, B.one, n5 & n6 & mm2);
            unsigned c = X[t] & kOClear;
            if (CLAMP) c = __vminu2(c, kOInf2);
            unsigned val = __viaddmin_u16x2(c, o_mad(col, B.one, own), kOInf2 + own);
            if (t == 0 && start && u == 0) val &= 0xFFFF0000u;  // MMM at cost 0
            x[S.code[t]] = val;
            h[S.code[t]] = true;
          }
          o_pass<1>(x, h, go2, B.one);
          o_pass<3>(x, h, go2, B.one);
          o_pass<9>(x, h, go2, B.one);
#pragma unroll
          for (int t = 0; t < kP3States; ++t) Tp[t] = x[S.code[t]];
          if (u == cap) endv = Tp[0];  // MMM opens nothing: the cell's least state
          row_out[(s + u) * 32] =
              make_uint4(o_prmt(Tp[R.t[1][0]], Tp[R.t[1][1]], 0x7632),
                         o_prmt(Tp[R.t[1][2]], Tp[R.t[1][3]], 0x7632),
                         o_prmt(Tp[R.t[5][0]], Tp[R.t[3][0]], 0x7632), Tp[R.t[7][0]]);
          if (lane == 31) {
            left_out[2 * (s + u)] = make_uint4(Tp[R.t[2][0]], Tp[R.t[2][1]], Tp[R.t[2][2]], Tp[R.t[2][3]]);
            left_out[2 * (s + u) + 1] = make_uint4(Tp[R.t[6][0]], U3, U7, 0);
          }
        }
        if (cap >= 0 && cap < 8) {
          unsigned *e = CL ? cg::this_cluster().map_shared_rank(&s_end, 0) : &s_end;
          *e = (na & 1) ? endv >> 16 : endv & 0xFFFFu;
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (CL) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    bar();
    if (rank == 0 && warp == 0) {
      // nibble st of cell (x, y, z): the state before st's column
      auto nib = [&](int x, int y, int z, int st) -> int {
        const int s = (y & 31) + z + (x & 1);
        const unsigned *p = reinterpret_cast<const unsigned *>(
            dir + (((int64_t)(x >> 1) * NB + (y >> 5)) * NS + s) * 32 + (y & 31));
        return (int)(__ldcg(p + (st >> 2)) >> (16 * (x & 1) + 4 * (st & 3))) & 15;
      };
      const unsigned e = s_end;
      // an optimum of 0xC000 / 16 or more reached the clamp: redo in 32 bits
      if ((e >= 0xC000u || !p3_walk_choices(A, c_p3o, i, lane, (int)(e >> 4), (int)(e & 15), nib)) &&
          lane == 0)
        atomicOr(A.err, 4);
    }
  }
}

constexpr size_t open_smem(int longest) {
  return (size_t)kOpenWarps * 2 * 8 * (32 + 2) * 16 + 2 * ((size_t)longest + 40 + 48);
}

}  // namespace

P3OpenPlan p3_open_plan(int64_t la, int64_t lb, int64_t lc) {
  const int64_t NS = (lc + 32 + 7) & ~(int64_t)7, NR = (la + 1) / 2, NB = (lb + 31) / 32;
  return {kOpenRing * NB * NS * 512 + NR * NB * NS * 32, NR * NB * NS * 512};
}

int p3_open_warps() { return kOpenWarps; }

namespace {

// A cluster's blocks get an SM each: two on one would halve its issue rate.
// (The request is the same for every length the entry points take.)
constexpr size_t kOpenClusterSmem = 116 * 1024;

cudaLaunchConfig_t open_config(int blocks, int csize, int longest, cudaLaunchAttribute *at,
                               cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)csize;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(blocks * csize));
  cfg.blockDim = dim3(32 * kOpenWarps);
  cfg.dynamicSmemBytes = csize > 1 ? kOpenClusterSmem : open_smem(longest);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = csize > 1 ? 1 : 0;
  return cfg;
}

}  // namespace

int p3_open_clusters(int csize) {
  static std::atomic<int> cache[64][9];
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int> &c = cache[dev & 63][csize];
  if (c.load() == 0) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = open_config(1, csize, 1, &at, nullptr);
    int n = 0;
    if (cudaFuncSetAttribute(k_p3_open<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)cfg.dynamicSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, k_p3_open<true, false>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    c.store(n > 0 ? n : -1);
  }
  return std::max(c.load(), 0);
}

int launch_p3_open(const P3Args &A, bool clamp, int longest, int blocks, int csize, uint8_t *plane,
                   int64_t plane_stride, uint8_t *dir, int64_t dir_stride, cudaStream_t st) {
  const OpenArgs B = {A, plane, plane_stride, dir, dir_stride, 1u, 16u, ~0u};
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = open_config(blocks, csize, longest, &at, st);
  auto kern = csize > 1 ? (clamp ? k_p3_open<true, true> : k_p3_open<true, false>)
                        : (clamp ? k_p3_open<false, true> : k_p3_open<false, false>);
  // the same request for every batch (one value per kernel and device, which a
  // thread with shorter sequences would lower under another's launch)
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(csize > 1 ? kOpenClusterSmem : open_smem(kP3MaxLen)));
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_p3_open)");
  ProfScope ps("p3", st);
  e = cudaLaunchKernelEx(&cfg, kern, B);
  return e != cudaSuccess ? cuda_fail(e, "k_p3_open") : POYD_OK;
}

}  // namespace poyd
