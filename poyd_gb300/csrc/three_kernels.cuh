// Shared by the three-sequence kernels (three.cu, three_linear.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "poyd_internal.h"

namespace poyd {

constexpr int kP3States = 16;
constexpr int kP3MaxLen = 4096;  // elements of a sequence that the entry points take

// Powell's column states (ukkCommon.c:206-262): per sequence match (M),
// delete (D) or insert (I), at least one M and at most one I, numbered in
// increasing order of x0 + 3 x1 + 9 x2 (M 0, D 1, I 2), MMM first.  A
// state without I consumes a character of each M sequence; a state with I
// consumes one of the I sequence only.  ngo[s][t] counts the gap openings
// of a step from s to t (ukkCommon.c:263-290): the sequences in D or I in
// t that were not in that same state in s.
struct P3States {
  int code[kP3States], adv[kP3States], ins[kP3States], ndel[kP3States];
  int ngo[kP3States][kP3States];
};

__host__ __device__ constexpr P3States p3_states() {
  P3States S{};
  int n = 0;
  for (int c = 0; c < 27; ++c) {
    const int x0 = c % 3, x1 = c / 3 % 3, x2 = c / 9 % 3;
    const int nm = (x0 == 0) + (x1 == 0) + (x2 == 0);
    const int ni = (x0 == 2) + (x1 == 2) + (x2 == 2);
    if (nm == 0 || ni > 1) continue;
    S.code[n] = c;
    S.ins[n] = ni;
    S.ndel[n] = 3 - nm - ni;
    S.adv[n] = ni ? ((x0 == 2) | (x1 == 2) << 1 | (x2 == 2) << 2)
                  : ((x0 == 0) | (x1 == 0) << 1 | (x2 == 0) << 2);
    ++n;
  }
  for (int s = 0; s < kP3States; ++s)
    for (int t = 0; t < kP3States; ++t) {
      int k = 0, cs = S.code[s], ct = S.code[t];
      for (int q = 0; q < 3; ++q, cs /= 3, ct /= 3)
        if (ct % 3 != 0 && ct % 3 != cs % 3) ++k;
      S.ngo[s][t] = k;
    }
  return S;
}

struct P3Args {
  int n, mode;            // mode 1: readjust_3d's early returns and changed flags
  const uint8_t *seq;
  const int64_t *off[4];  // a, b, c; m (mode 1)
  const int32_t *len[4];
  int32_t *cost;
  uint8_t *out;
  const int64_t *out_off;
  int32_t *out_len;
  int32_t *changed;
  const int32_t *order;
  int32_t *counter;
  int32_t *err;
  int32_t *ring;
  int64_t ring_stride;    // int32 per block
  uint64_t *dir;
  int64_t dir_stride;     // words per block
  int mm, go, ge, gap, has_med, smax;
  uint8_t med[128];       // Three_D.median of (x, y, z) over A C G T gap, 25 x + 5 y + z
};

__device__ __forceinline__ int p3_code(int x) {  // copySequence: lowest of A C G T
  return (x & 1) ? 1 : (x & 2) ? 2 : (x & 4) ? 4 : (x & 8) ? 8 : 0;
}
__device__ __forceinline__ int p3_ix(int x) { return __ffs(x) - 1; }  // 1 2 4 8 16 -> 0..4

// What every kernel does with a triple before its DP, by all `nthr` threads
// of the block: readjust_3d's early returns (sequence.ml:1118-1129; is_empty
// is sequence.ml:442-450) and the characters Powell's code aligns
// (copySequence, ukkCommon.c:84-105) through put(q, x, code) for x >= 1.
// Returns false when the triple is done (early return, or an element without
// a base); `lead` blocks write its outputs.
template <class Put>
__device__ __forceinline__ bool p3_begin(const P3Args &A, int i, bool lead, int tid, int nthr,
                                         Put put) {
  const int l[3] = {A.len[0][i], A.len[1][i], A.len[2][i]};
  const uint8_t *src[3] = {A.seq + A.off[0][i], A.seq + A.off[1][i], A.seq + A.off[2][i]};
  const int cap = (l[0] + l[1] + l[2] + 3) & ~3;
  uint8_t *o = A.out + A.out_off[i];
  if (A.mode == 1) {
    const int lm = A.len[3][i];
    const uint8_t *m = A.seq + A.off[3][i];
    int keep = 0;  // 1 m, 2 b, 3 a, 4 c
    if (l[0] == l[1] && lm == l[2] && l[0] == lm) {
      keep = 1;
    } else {
      bool e[3] = {true, true, true};
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        bool all = true;
        for (int x = tid; x < l[q]; x += nthr) all &= src[q][x] == A.gap;
        e[q] = __syncthreads_and(all);
      }
      keep = (e[0] && !e[1]) ? 2 : (e[1] && !e[0]) ? 3 : e[2] ? 4 : 0;
    }
    if (keep) {
      const uint8_t *k = keep == 1 ? m : keep == 2 ? src[1] : keep == 3 ? src[0] : src[2];
      const int lk = keep == 1 ? lm : keep == 2 ? l[1] : keep == 3 ? l[0] : l[2];
      bool diff = lk != lm;
      for (int x = tid; x < lk; x += nthr) {
        if (lead) o[4 * cap - lk + x] = k[x];
        if (lk == lm) diff |= k[x] != m[x];
      }
      diff = __syncthreads_or(diff);
      if (lead && tid == 0) {
        A.cost[i] = 0;
        A.out_len[2 * i] = 0;
        A.out_len[2 * i + 1] = lk;
        A.changed[i] = diff ? 1 : 0;
      }
      return false;
    }
  }
  bool bad = false;
#pragma unroll
  for (int q = 0; q < 3; ++q)
    for (int x = 1 + tid; x < l[q]; x += nthr) {
      const int c = p3_code(src[q][x]);
      bad |= c == 0;
      put(q, x, c);
    }
  if (__syncthreads_or(bad)) {
    if (lead && tid == 0) {
      A.cost[i] = -1;
      A.out_len[2 * i] = -1;
      A.out_len[2 * i + 1] = -1;
      if (A.mode == 1) A.changed[i] = 0;
      atomicOr(A.err, 1);
    }
    return false;
  }
  return true;
}

// Column cost of state t (alignmentCost, ukkCommon.c:345-391) for the
// consumed characters (one bit each; 0 or 16: none).
__device__ __forceinline__ int p3_col(const P3States &S, const P3Args &A, int t, int c0, int c1,
                                      int c2) {
  if (S.ins[t]) return A.ge;
  const int ch = (c0 | c1 | c2) & 15;
  return A.mm * (__popc(ch) - 1) + S.ndel[t] * A.ge;
}

// The outputs of one triple written from the end by one warp, 32 columns at a
// time: the walk tells which columns, this writes them.
struct P3Writer {
  const P3Args &A;
  const P3States &S;
  int i, lane, cap;
  const uint8_t *sq[3];
  uint8_t *o;
  int n, nm, cost;

  __device__ __forceinline__ P3Writer(const P3Args &A_, const P3States &S_, int i_, int lane_)
      : A(A_), S(S_), i(i_), lane(lane_), n(0), nm(0), cost(0) {
    for (int q = 0; q < 3; ++q) sq[q] = A.seq + A.off[q][i];
    cap = (A.len[0][i] + A.len[1][i] + A.len[2][i] + 3) & ~3;
    o = A.out + A.out_off[i];
  }
  // column n + lane of cell (x, y, z) in state st on the lanes with `writes`
  // (lanes 0 .. count - 1)
  __device__ __forceinline__ void put(bool writes, int count, int st, int x, int y, int z) {
    int md = A.gap, col = 0;
    if (writes) {
      const int ad = S.adv[st];
      const int ca = (ad & 1) ? p3_code(sq[0][x]) : 16, cb = (ad & 2) ? p3_code(sq[1][y]) : 16,
                cc = (ad & 4) ? p3_code(sq[2][z]) : 16;
      col = p3_col(S, A, st, ca, cb, cc);
      md = A.med[25 * p3_ix(ca) + 5 * p3_ix(cb) + p3_ix(cc)];
      const int p = cap - 1 - (n + lane);
      o[p] = (uint8_t)ca;
      o[cap + p] = (uint8_t)cb;
      o[2 * cap + p] = (uint8_t)cc;
    }
    const bool keep = writes && A.has_med && md != A.gap;
    const unsigned kb = __ballot_sync(0xffffffffu, keep);
    if (keep) o[4 * cap - 1 - (nm + __popc(kb & ((1u << lane) - 1u)))] = (uint8_t)md;
    cost += __reduce_add_sync(0xffffffffu, col);
    n += count;
    nm += __popc(kb);
  }
  // the leading gap column (printTraceBack, ukk.checkp.c), lengths, cost and
  // changed flag
  __device__ __forceinline__ void finish(int total) {
    ++n;
    if (lane == 0) {
      o[cap - n] = o[2 * cap - n] = o[3 * cap - n] = 16;
      if (A.has_med) o[4 * cap - 1 - nm] = (uint8_t)A.gap;
    }
    if (A.has_med) ++nm;
    __syncwarp();
    bool diff = false;
    if (A.mode == 1) {
      const int lm = A.len[3][i];
      const uint8_t *m = A.seq + A.off[3][i];
      diff = nm != lm;
      if (!diff)
        for (int x = lane; x < lm; x += 32) diff |= o[4 * cap - nm + x] != m[x];
      diff = __any_sync(0xffffffffu, diff);
    }
    if (lane == 0) {
      A.cost[i] = total;
      A.out_len[2 * i] = n;
      A.out_len[2 * i + 1] = A.has_med ? nm : 0;
      if (A.mode == 1) A.changed[i] = diff ? 1 : 0;
    }
  }
};

// The walk of the zero-opening kernel, by one warp: nib(a, b, c) is a cell's
// own best state.  Most columns are MMM, so lane k reads the cell k columns up
// the diagonal; the run up to the first other state and that state's column
// are taken at once.  Returns false when the path left the cube or its cost
// is not exact (>= most).
template <class Nib>
__device__ __forceinline__ bool p3_walk_states(const P3Args &A, const P3States &S, int i, int lane,
                                               int most, Nib nib) {
  P3Writer w(A, S, i, lane);
  int a = A.len[0][i] - 1, b = A.len[1][i] - 1, c = A.len[2][i] - 1;
  while (a | b | c) {
    const int x = a - lane, y = b - lane, z = c - lane;
    const bool in = x >= 0 && y >= 0 && z >= 0 && (x | y | z);
    const int st = in ? nib(x, y, z) : 0;
    // a state this cell cannot be in ends the walk (the path is not exact)
    const int ad = S.adv[st];
    const bool ok = in && !((ad & 1) > x || (ad >> 1 & 1) > y || (ad >> 2 & 1) > z);
    const unsigned stop = __ballot_sync(0xffffffffu, !ok || st != 0);
    const int f = stop ? __ffs(stop) - 1 : 32;  // lanes below f: MMM columns
    const bool step_f = f < 32 && (__ballot_sync(0xffffffffu, ok) >> (f & 31) & 1);
    const int in_f = __shfl_sync(0xffffffffu, (int)in, f & 31);
    if (f < 32 && !step_f && (f == 0 || in_f)) return false;
    const int ad_f = step_f ? __shfl_sync(0xffffffffu, ad, f & 31) : 0;
    w.put(lane < f + step_f, f + step_f, st, x, y, z);
    a -= f + (ad_f & 1);
    b -= f + (ad_f >> 1 & 1);
    c -= f + (ad_f >> 2 & 1);
  }
  if (w.cost >= most) return false;
  w.finish(w.cost);
  return true;
}

// The walk of the kernels with openings: nib(a, b, c, st) is the state before
// a column in state st at the cell; the walk starts in state st with the
// optimum `total`.  A run of MMM columns ends after the one whose previous
// state is another.
template <class Nib>
__device__ __forceinline__ bool p3_walk_choices(const P3Args &A, const P3States &S, int i, int lane,
                                                int total, int st, Nib nib) {
  P3Writer w(A, S, i, lane);
  int a = A.len[0][i] - 1, b = A.len[1][i] - 1, c = A.len[2][i] - 1;
  while (a | b | c) {
    const int ad = S.adv[st];
    if ((ad & 1) > a || (ad >> 1 & 1) > b || (ad >> 2 & 1) > c) return false;
    if (st != 0) {
      const int prev = nib(a, b, c, st);
      w.put(lane == 0, 1, st, a, b, c);
      a -= ad & 1;
      b -= ad >> 1 & 1;
      c -= ad >> 2 & 1;
      st = prev;
      continue;
    }
    const int x = a - lane, y = b - lane, z = c - lane;
    const bool in = x > 0 && y > 0 && z > 0;
    const int prev = in ? nib(x, y, z, 0) : 0;
    const unsigned stop = __ballot_sync(0xffffffffu, !in || prev != 0);
    const int f = stop ? __ffs(stop) - 1 : 32;
    const bool step_f = f < 32 && (__ballot_sync(0xffffffffu, in) >> (f & 31) & 1);
    st = step_f ? __shfl_sync(0xffffffffu, prev, f & 31) : 0;
    w.put(lane < f + step_f, f + step_f, 0, x, y, z);
    a -= f + step_f;
    b -= f + step_f;
    c -= f + step_f;
  }
  w.finish(total);
  return true;
}

// The kernel for go = 0 (three_linear.cu): scratch bytes per block for
// triples of at most (la, lb, lc) elements, the warps of a block for a batch
// whose longest sequence has `longest` elements, and the launch.
struct P3LinearPlan {
  int64_t plane, dir;  // bytes per block: strip boundaries, choices
};
P3LinearPlan p3_linear_plan(int64_t la, int64_t lb, int64_t lc);
int p3_linear_blocks(int warps, int longest);  // resident blocks of the device
// Warp steps of a triple in all, and of the longest of its `warps` warps.
int64_t p3_linear_steps(int64_t la, int64_t lb, int64_t lc);
int64_t p3_linear_chain(int64_t la, int64_t lb, int64_t lc, int warps);
int launch_p3_linear(const P3Args &A, int warps, int longest, int blocks, uint8_t *plane,
                     int64_t plane_stride, uint8_t *dir, int64_t dir_stride, cudaStream_t st);
constexpr int kP3LinLag = 48;  // steps between consecutive strips

// The 16-bit kernel with openings (three_open.cu): scratch bytes per triple in
// flight, warps of a block, and the launch of `blocks` clusters of csize.
struct P3OpenPlan {
  int64_t plane, dir;
};
P3OpenPlan p3_open_plan(int64_t la, int64_t lb, int64_t lc);
int p3_open_warps();
int p3_open_clusters(int csize);  // clusters of csize blocks the device holds at once
int launch_p3_open(const P3Args &A, bool clamp, int longest, int blocks, int csize, uint8_t *plane,
                   int64_t plane_stride, uint8_t *dir, int64_t dir_stride, cudaStream_t st);

}  // namespace poyd
