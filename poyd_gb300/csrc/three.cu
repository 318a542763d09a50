// Three-sequence alignment of the Iterative (ThreeD) cost mode.
//
// Sequence.Align.readjust_3d (sequence.ml:1117-1140) re-estimates a node's
// median from its two children and its parent with align_3_powell_inter
// (sequence.ml:1089-1115), which aligns the three sequences with
// powell_3D_align (ukkCommon.c:111-143): Powell's three-way generalisation
// of Ukkonen's algorithm over 16 column states, with check-pointing
// (ukk.checkp.c).  Its cost is the optimum of a fixed cost model
// (alignmentCost, ukkCommon.c:345-391), which does not depend on how the
// optimum is searched.  Each triple is one dynamic program over the full
// (la x lb x lc) cube, one cell's states from its seven neighbours', by one of
// three kernels:
//   * three_linear.cu: no gap openings (go = 0, the linear model), 16-bit
//     values, one optimum per cell;
//   * three_open.cu: gap openings, 16-bit values;
//   * k_p3 (here): 32-bit values, for batches whose costs may not fit 16 bits,
//     swept by hyperplanes h = i + j + k (a cell depends only on the three
//     hyperplanes before it): one block per triple, persistent over a
//     largest-first queue; a warp takes a row (fixed i) of the hyperplane, a
//     lane one cell of it.  Every state reads one neighbour cell (the one its
//     column consumes from); values are stored x16 with a state number in the
//     low 4 bits, so that one add-min per (previous, next) state pair keeps
//     the least cost and, on ties, the lowest-numbered previous state.  The
//     last four hyperplanes' values are a ring in global memory
//     ([h & 3][i][j][state]); the 16 choices of a cell (4 bits each) one
//     64-bit word of a per-triple cube laid out [i][j + k][j] so that a
//     hyperplane's cells of one i are contiguous.
// One warp then walks the choices back (three_kernels.cuh) and writes the
// three aligned rows and the column medians (Cost_matrix.Three_D.median)
// right-aligned into the triple's slot.
// Among equally cheap alignments the walk keeps the lowest-numbered final
// state and at every column the lowest-numbered previous state; Powell's
// recursion may return another of the optimal alignments.
#include <algorithm>
#include <cstring>
#include <vector>

#include "three_kernels.cuh"

#define CK3(call)                                         \
  do {                                                    \
    cudaError_t e_ = (call);                              \
    if (e_ != cudaSuccess) return cuda_fail(e_, #call);   \
  } while (0)

namespace poyd {

constexpr int kP3Threads = 256;
constexpr int kP3Inf = 1 << 30;      // x16 domain

// The same tables for indices known only at run time (traceback, table
// setup): constant memory rather than a local copy.
__constant__ P3States c_p3 = p3_states();

// Offset of the (j + k = s) row in an i-slice of the choice cube:
// the sum over s' < s of the row lengths min(nb, s') - max(0, s' - nc) + 1.
__device__ __forceinline__ int64_t p3_soff(int s, int nb, int nc) {
  int64_t f;
  if (s <= nb + 1) f = (int64_t)s * (s + 1) / 2;
  else f = (int64_t)(nb + 1) * (nb + 2) / 2 + (int64_t)(s - nb - 1) * (nb + 1);
  if (s > nc + 1) {
    const int64_t m = s - nc - 1;
    f -= m * (m + 1) / 2;
  }
  return f;
}

// One cell (a, b, c) of hyperplane h: its 16 values (x16, into the ring)
// and its 64-bit choice word (returned).
__device__ __forceinline__ uint64_t p3_cell(int32_t *ring, int64_t pl, int nb, int h, int a,
                                            int b, int c, const int *g16, const int *col16) {
  constexpr P3States S = p3_states();
  int best[kP3States];
#pragma unroll
  for (int t = 0; t < kP3States; ++t) best[t] = kP3Inf;
#pragma unroll
  for (int d = 1; d < 8; ++d) {  // the neighbour cell one column of step d back
    const int da = d & 1, db = d >> 1 & 1, dc = d >> 2 & 1;
    if (a < da || b < db || c < dc) continue;
    const int hs = h - da - db - dc;
    const int4 *p = reinterpret_cast<const int4 *>(
        ring + ((int64_t)(hs & 3) * pl + (int64_t)(a - da) * (nb + 1) + (b - db)) * kP3States);
    int w[kP3States];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int4 u = p[q];
      w[4 * q] = u.x + 4 * q;  // the previous state in the low bits
      w[4 * q + 1] = u.y + 4 * q + 1;
      w[4 * q + 2] = u.z + 4 * q + 2;
      w[4 * q + 3] = u.w + 4 * q + 3;
    }
#pragma unroll
    for (int t = 0; t < kP3States; ++t) {
      if (S.adv[t] != d) continue;
#pragma unroll
      for (int s = 0; s < kP3States; ++s) best[t] = __viaddmin_s32(w[s], g16[S.ngo[s][t]], best[t]);
    }
  }
  int4 *o = reinterpret_cast<int4 *>(
      ring + ((int64_t)(h & 3) * pl + (int64_t)a * (nb + 1) + b) * kP3States);
  uint64_t word = 0;
  int v[kP3States];
#pragma unroll
  for (int t = 0; t < kP3States; ++t) {
    const bool fin = best[t] < kP3Inf;
    // an I column costs one extension; otherwise one per D plus the
    // mismatches of the matched characters
    const int col = S.ins[t] ? g16[4] : col16[S.adv[t]] + S.ndel[t] * g16[4];
    v[t] = fin ? (best[t] & ~15) + col : kP3Inf;
    word |= (uint64_t)(fin ? best[t] & 15 : 0) << (4 * t);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = make_int4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  return word;
}

__global__ void __launch_bounds__(kP3Threads) k_p3(const __grid_constant__ P3Args A) {
  extern __shared__ uint8_t p3_sm[];
  __shared__ int s_job;
  uint8_t *sq[3] = {p3_sm, p3_sm + A.smax, p3_sm + 2 * A.smax};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kP3Threads / 32;
  // x16 costs: g16[k] = k gap openings, g16[4] = one extension
  const int g16[5] = {0, 16 * A.go, 32 * A.go, 48 * A.go, 16 * A.ge};
  int32_t *ring = A.ring + blockIdx.x * A.ring_stride;
  uint64_t *dir = A.dir + blockIdx.x * A.dir_stride;

  for (;;) {
    __syncthreads();
    if (tid == 0) s_job = atomicAdd(A.counter, 1);
    __syncthreads();
    if (s_job >= A.n) break;
    const int i = A.order[s_job];
    const int la = A.len[0][i], lb = A.len[1][i], lc = A.len[2][i];
    if (!p3_begin(A, i, true, tid, kP3Threads,
                  [&](int q, int x, int c) { sq[q][x] = (uint8_t)c; }))
      continue;

    const int na = la - 1, nb = lb - 1, nc = lc - 1, H = na + nb + nc;
    const int64_t pl = (int64_t)(na + 1) * (nb + 1);  // ring plane (cells)
    const int64_t bcs = (int64_t)(nb + 1) * (nc + 1); // choice-cube i-slice
    for (int h = 0; h <= H; ++h) {
      const int a_lo = max(0, h - nb - nc), a_hi = min(na, h);
      for (int a = a_lo + warp; a <= a_hi; a += kWarps) {  // a warp per row
        const int s = h - a, blo = max(0, s - nc), bhi = min(nb, s);
        const int64_t drow = (int64_t)a * bcs + p3_soff(s, nb, nc) - blo;
        for (int b = blo + lane; b <= bhi; b += 32) {
          const int c = s - b;
          uint64_t word = 0;
          if (h == 0) {  // the start: MMM at cost 0
            int4 *r = reinterpret_cast<int4 *>(ring);
            r[0] = make_int4(0, kP3Inf, kP3Inf, kP3Inf);
            for (int q = 1; q < 4; ++q) r[q] = make_int4(kP3Inf, kP3Inf, kP3Inf, kP3Inf);
          } else {
            // alignmentCost's mismatches (ukkCommon.c:381-389), x16, by the
            // sequences a column consumes: mm per extra distinct character
            const int x0 = a ? sq[0][a] : 0, x1 = b ? sq[1][b] : 0, x2 = c ? sq[2][c] : 0;
            int col16[8];
            col16[0] = 0;
#pragma unroll
            for (int d = 1; d < 8; ++d) {
              const int ch = ((d & 1) ? x0 : 0) | ((d & 2) ? x1 : 0) | ((d & 4) ? x2 : 0);
              col16[d] = 16 * A.mm * (__popc(ch) - 1);
            }
            word = p3_cell(ring, pl, nb, h, a, b, c, g16, col16);
          }
          dir[drow + b] = word;
        }
      }
      __syncthreads();
    }
    if (warp == 0) {
      const int32_t *f = ring + ((int64_t)(H & 3) * pl + (int64_t)na * (nb + 1) + nb) * kP3States;
      int best = kP3Inf, st = 0;
      for (int s = 0; s < kP3States; ++s)
        if (f[s] < best) best = f[s], st = s;
      auto nib = [&](int x, int y, int z, int t) -> int {
        const int s = y + z;
        return (int)(dir[(int64_t)x * bcs + p3_soff(s, nb, nc) + (y - max(0, s - nc))] >> (4 * t)) & 15;
      };
      if (best >= kP3Inf || !p3_walk_choices(A, c_p3, i, lane, best >> 4, st, nib)) {
        if (lane == 0) {  // cannot happen for a finite optimum; kept as a guard
          atomicOr(A.err, 2);
          A.cost[i] = A.out_len[2 * i] = A.out_len[2 * i + 1] = -1;
          if (A.mode == 1) A.changed[i] = 1;
        }
      }
    }
  }
}

// Cost_matrix.Three_D.of_two_dim_comb (cost_matrix.ml:803-851): the median
// of (i, j, k) is the lowest single state l with the least
// cost[l][i] + cost[l][j] + cost[l][k]; the gap takes part only for metric
// matrices or when two of i, j, k hold it.  The reference seeds each entry
// with OCaml's max_int, which fits a C int on a 32-bit OCaml only (on a
// 64-bit one it truncates to -1 and no entry is ever set); this follows the
// 32-bit reading.
static uint8_t median3_of(const poyd_cm *cm, int i, int j, int k) {
  int64_t best = INT64_MAX;
  int med = 0;
  for (int l = 0; l < cm->lcm; ++l) {
    const int x = 1 << l;
    const int shared = ((i & x) != 0) + ((j & x) != 0) + ((k & x) != 0);
    int64_t c = INT64_MAX;
    if (cm->is_metric || shared >= 2 || x != cm->gap)
      c = (int64_t)cm->cost[(x << 5) + i] + cm->cost[(x << 5) + j] + cm->cost[(x << 5) + k];
    if (c < best) {
      best = c;
      med = x;
    } else if (c == best) {
      med |= x;
    }
  }
  return (uint8_t)(med & -med);
}
static void median3_table(const poyd_cm *cm, uint8_t *tab) {
  std::memset(tab, 0, 32768);
  for (int i = 1; i < 32; ++i)
    for (int j = 1; j < 32; ++j)
      for (int k = 1; k < 32; ++k) tab[(i << 10) | (j << 5) | k] = median3_of(cm, i, j, k);
}

// The lengths side by side, for one copy to the host.
__global__ void k_p3_lens(int n, const int32_t *a, const int32_t *b, const int32_t *c,
                          const int32_t *d, int32_t *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = a[i];
  out[n + i] = b[i];
  out[2 * (int64_t)n + i] = c[i];
  if (d) out[3 * (int64_t)n + i] = d[i];
}

// Host side shared by the two batched entry points.
static int p3_run(int mode, int32_t n, const uint8_t *seq, const int64_t *const off[4],
                  const int32_t *const len[4], int mm, int go, int ge, int gap,
                  const uint8_t *median3, const poyd_cm *median_cm, int32_t *cost, uint8_t *out,
                  const int64_t *out_off, int32_t *out_len, int32_t *changed, cudaStream_t st) {
  if (n < 0) return fail(POYD_EINVAL, "three-sequence batch: n < 0");
  if (n == 0) return POYD_OK;
  if (!seq || !cost || !out || !out_off || !out_len || (mode == 1 && !changed))
    return fail(POYD_EINVAL, "three-sequence batch: null argument");
  if (mm <= 0 || go < 0 || ge <= 0)
    return fail(POYD_EINVAL, "powell_3D_align needs mm > 0, go >= 0, ge > 0 (ukkCommon.c:130)");
  const int nq = mode == 1 ? 4 : 3;
  for (int q = 0; q < nq; ++q)
    if (!off[q] || !len[q]) return fail(POYD_EINVAL, "three-sequence batch: null argument");
  Workspace *w = workspace(st);
  // the lengths to the host, in one copy
  int32_t *dlen = (int32_t *)ws_buffer(w, WS_P3_LENS, sizeof(int32_t) * (size_t)n * nq);
  if (!dlen) return fail(POYD_ENOMEM, "three-sequence workspace");
  k_p3_lens<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, len[0], len[1], len[2],
                                                        nq == 4 ? len[3] : nullptr, dlen);
  CK3(cudaGetLastError());
  std::vector<int32_t> all_len((size_t)n * nq);
  CK3(cudaMemcpyAsync(all_len.data(), dlen, sizeof(int32_t) * (size_t)n * nq, cudaMemcpyDeviceToHost, st));
  CK3(cudaStreamSynchronize(st));
  const int32_t *hl[4];
  for (int q = 0; q < 4; ++q) hl[q] = all_len.data() + (size_t)n * std::min(q, nq - 1);
  int64_t ring_max = 0, dir_max = 0, lin_plane = 0, lin_dir = 0, lin_steps = 0;
  int64_t open_plane = 0, open_dir = 0;
  int smax = 16, max_b = 1;
  std::vector<int64_t> work(n);
  const int64_t step_max = 2LL * go + 2LL * ge + 2LL * mm;
  for (int32_t i = 0; i < n; ++i) {
    const int64_t la = hl[0][i], lb = hl[1][i], lc = hl[2][i];
    if (la < 1 || lb < 1 || lc < 1 || (mode == 1 && hl[3][i] < 0))
      return fail(POYD_EINVAL, "triple %d: every sequence holds at least its leading gap", i);
    if (la > kP3MaxLen || lb > kP3MaxLen || lc > kP3MaxLen)
      return fail(POYD_ERANGE, "triple %d: sequences longer than %d", i, kP3MaxLen);
    if ((la + lb + lc) * step_max * 16 >= kP3Inf / 2)
      return fail(POYD_ERANGE, "triple %d: costs could reach the DP's infinity", i);
    ring_max = std::max(ring_max, 4 * la * lb * kP3States);
    dir_max = std::max(dir_max, la * lb * lc);
    smax = std::max<int>(smax, (int)std::max(la, std::max(lb, lc)));
    work[i] = la * lb * lc;
    const P3LinearPlan lp = p3_linear_plan(la, lb, lc);
    lin_steps += p3_linear_steps(la, lb, lc);
    lin_plane = std::max(lin_plane, lp.plane);
    lin_dir = std::max(lin_dir, lp.dir);
    const P3OpenPlan op = p3_open_plan(la, lb, lc);
    open_plane = std::max(open_plane, op.plane);
    open_dir = std::max(open_dir, op.dir);
    max_b = std::max(max_b, (int)lb);
  }
  const int longest = smax;
  smax = (smax + 15) & ~15;
  std::vector<int32_t> order;
  longest_first(work, order);

  int dev = 0, sms = 0;
  CK3(cudaGetDevice(&dev));
  CK3(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // Blocks of a launch whose buffers take ring + dir bytes each.  The choices
  // dominate: one set per resident block, sized for the largest triple; by default
  // at most 60 % of the free memory, 120 GiB (asked for only where the buffers do
  // not hold the launch already).
  auto fit = [&](int64_t want, int64_t ring, int64_t dir) -> int64_t {
    int64_t budget;
    if (const char *e = getenv("POYD_P3_BUDGET_MB")) {
      budget = std::max<int64_t>(1, atoll(e)) << 20;
    } else {
      if ((size_t)(ring * want) <= ws_size(w, WS_P3_RING) && (size_t)(dir * want) <= ws_size(w, WS_P3_DIR))
        return want;
      size_t fr = 0, tot = 0;
      if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return 1;
      budget = std::min<int64_t>((int64_t)(fr * 0.6), 120LL << 30);
    }
    return std::min(want, std::max<int64_t>(1, budget / (ring + dir)));
  };
  int32_t *meta = (int32_t *)ws_buffer(w, WS_P3_META, sizeof(int32_t) * ((size_t)n + 4));
  if (!meta) return fail(POYD_ENOMEM, "three-sequence workspace");
  order.push_back(0);  // counter
  order.push_back(0);  // err
  CK3(cudaMemcpyAsync(meta, order.data(), sizeof(int32_t) * ((size_t)n + 2), cudaMemcpyHostToDevice, st));

  P3Args A;
  std::memset(&A, 0, sizeof(A));
  A.n = n;
  A.mode = mode;
  A.seq = seq;
  for (int q = 0; q < nq; ++q) {
    A.off[q] = off[q];
    A.len[q] = len[q];
  }
  A.cost = cost;
  A.out = out;
  A.out_off = out_off;
  A.out_len = out_len;
  A.changed = changed;
  A.order = meta;
  A.counter = meta + n;
  A.err = meta + n + 1;
  A.mm = mm;
  A.go = go;
  A.ge = ge;
  A.gap = gap;
  A.has_med = median3 || median_cm ? 1 : 0;
  {
    static const int st5[5] = {1, 2, 4, 8, 16};
    for (int x = 0; x < 5; ++x)
      for (int y = 0; y < 5; ++y)
        for (int z = 0; z < 5; ++z)
          A.med[25 * x + 5 * y + z] =
              median_cm ? median3_of(median_cm, st5[x], st5[y], st5[z])
              : median3 ? median3[(st5[x] << 10) | (st5[y] << 5) | st5[z]] : (uint8_t)gap;
  }
  A.smax = smax;
  // the launch's error bits; bit 2: an optimum reached the 16-bit clamp, the
  // batch is redone in 32 bits
  auto finish = [&](bool *redo) -> int {
    int32_t herr = 0;
    CK3(cudaGetLastError());
    CK3(cudaMemcpyAsync(&herr, A.err, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK3(cudaStreamSynchronize(st));
    *redo = false;
    if (herr & 1)
      return fail(POYD_EINVAL, "an element holds none of A, C, G, T (powell_3D_align fails, "
                               "ukkCommon.c:101): its triple has cost -1");
    if (herr & 2) return fail(POYD_ERANGE, "three-sequence traceback left the cube");
    if (!(herr & 4)) return POYD_OK;
    *redo = true;
    const int32_t zero2[2] = {0, 0};
    CK3(cudaMemcpyAsync(A.counter, zero2, sizeof(zero2), cudaMemcpyHostToDevice, st));
    return POYD_OK;
  };
  // 16-bit halves while every addend of a half stays below 0x4000
  // (openings, column costs)
  const char *pk = getenv("POYD_P3_PACKED");
  const bool packed = !(pk && pk[0] == '0') && 48LL * go + 15 < 0x4000 &&
                16LL * (2LL * mm + 3LL * ge) < 0x4000;
  if (packed && go == 0) {
    // Warps per triple: twice as many while the largest triple's own steps get
    // fewer by three tenths (its strips follow one another kP3LinLag steps apart,
    // so that a strip feeds steps / kP3LinLag warps; 20 triples of 150-200 bp, a
    // fifth fewer steps, take 1.15 ms with 4 warps and 1.37 with more) and its own
    // time, at four warps a scheduler, is more than three quarters of what the
    // whole batch's instructions take.
    // Up to two triples an SM, then twice as many where that costs no step: a
    // block an SM, whose waiting warps leave the others the issue slots.
    // Measured with 2, 4, 8 and 16 warps: 1,216 triples of 100-300 bp 17.6, 10.1,
    // 8.9 and 11.4 ms, of 200 bp 6.6, 6.1, 9.0 and 10.7; 304 of 100-300 bp 6.5,
    // 5.4, 5.3 and 3.1.
    const int big = order[0];
    const int64_t bl[3] = {hl[0][big], hl[1][big], hl[2][big]};
    auto chain = [&](int w) { return p3_linear_chain(bl[0], bl[1], bl[2], w); };
    const double batch = 280.0 * (double)lin_steps / (4.0 * sms);
    int warps = 1;
    while (warps < 16 && 10 * chain(2 * warps) <= 7 * chain(warps) &&
           1100.0 * (double)chain(warps) > 0.75 * batch)
      warps *= 2;
    if (n <= 2 * sms && warps == 8 && chain(16) <= chain(8)) warps = 16;
    const int blocks = (int)fit(std::min<int64_t>(n, p3_linear_blocks(warps, longest)), lin_plane, lin_dir);
    uint8_t *plane = (uint8_t *)ws_buffer(w, WS_P3_RING, (size_t)(lin_plane * blocks));
    uint8_t *dirb = (uint8_t *)ws_buffer(w, WS_P3_DIR, (size_t)(lin_dir * blocks));
    if (!plane || !dirb) return fail(POYD_ENOMEM, "three-sequence workspace (%d blocks)", blocks);
    int rc = launch_p3_linear(A, warps, longest, blocks, plane, lin_plane, dirb, lin_dir, st);
    if (rc) return rc;
    bool redo = false;
    rc = finish(&redo);
    if (rc || !redo) return rc;
  } else if (packed) {
    // Small batches take a cluster of blocks per triple, an SM each: a triple
    // feeds (strips of b) x (steps of a task / the rows' lag) warps.  The
    // largest size of which the whole batch is resident at once (a cluster
    // sits in one GPC, whose SMs a size may not divide: 20 clusters of 6 ran
    // in two waves, 2.5 ms against 1.6 for one wave).
    // POYD_P3_CLUSTER=0: one block per triple.
    const int64_t useful = (int64_t)((max_b + 31) / 32) * ((longest + 40) / 32 + 1);
    const char *ce = getenv("POYD_P3_CLUSTER");
    int csize = ce && ce[0] == '0' ? 1 : (int)std::min<int64_t>(
        {8, (useful + p3_open_warps() - 1) / p3_open_warps(), std::max<int64_t>(1, sms / n)});
    while (csize > 1 && p3_open_clusters(csize) < n) --csize;
    int blocks = (int)fit(std::min<int64_t>(n, 2LL * sms), open_plane, open_dir);
    uint8_t *plane = (uint8_t *)ws_buffer(w, WS_P3_RING, (size_t)(open_plane * blocks));
    uint8_t *dirb = (uint8_t *)ws_buffer(w, WS_P3_DIR, (size_t)(open_dir * blocks));
    // Its strips of 32 want more memory than k_p3's cube (a sixteenth more, up to 32
    // times for a b of one element): what that can hold is not refused.
    if (plane && dirb) {
      // a sum of an opened value and a column cost may pass 16 bits: cut it off
      const bool clamp = 48LL * go + 16LL * (2LL * mm + 3LL * ge) + 31 >= 0x4000;
      int rc = launch_p3_open(A, clamp, longest, blocks, csize, plane, open_plane, dirb, open_dir, st);
      if (rc) return rc;
      bool redo = false;
      rc = finish(&redo);
      if (rc || !redo) return rc;
    }
  }
  const int64_t blocks = fit(std::min<int64_t>(n, 3LL * sms), ring_max * 4, dir_max * 8);
  A.ring = (int32_t *)ws_buffer(w, WS_P3_RING, (size_t)(ring_max * 4 * blocks));
  A.dir = (uint64_t *)ws_buffer(w, WS_P3_DIR, (size_t)(dir_max * 8 * blocks));
  if (!A.ring || !A.dir)
    return fail(POYD_ENOMEM, "three-sequence workspace (%lld blocks)", (long long)blocks);
  A.ring_stride = ring_max;
  A.dir_stride = dir_max;
  const size_t smem = 3 * (size_t)smax;
  {
    ProfScope ps("p3", st);
    k_p3<<<(unsigned)blocks, kP3Threads, smem, st>>>(A);
  }
  bool redo = false;
  return finish(&redo);
}

}  // namespace poyd

using namespace poyd;

extern "C" int poyd_cm_median3(const poyd_cm *cm, uint8_t *tab) {
  if (!cm || !tab) return fail(POYD_EINVAL, "poyd_cm_median3: null argument");
  if (!cm->combinations || cm->lcm < 1 || cm->lcm > 5)
    return fail(POYD_EUNSUP, "poyd_cm_median3: combination alphabets of at most 5 states");
  median3_table(cm, tab);
  return POYD_OK;
}

extern "C" int poyd_powell_3d_batch(int32_t n, const uint8_t *seq, const int64_t *a_off,
                                    const int32_t *a_len, const int64_t *b_off,
                                    const int32_t *b_len, const int64_t *c_off,
                                    const int32_t *c_len, int32_t mm, int32_t go, int32_t ge,
                                    const uint8_t *median3, int32_t *cost, uint8_t *out,
                                    const int64_t *out_off, int32_t *out_len, void *stream) {
  const int64_t *off[4] = {a_off, b_off, c_off, nullptr};
  const int32_t *len[4] = {a_len, b_len, c_len, nullptr};
  return p3_run(0, n, seq, off, len, mm, go, ge, 16, median3, nullptr, cost, out, out_off, out_len,
                nullptr, (cudaStream_t)stream);
}

extern "C" int poyd_readjust_3d_batch(const poyd_cm *cm, int32_t n, const uint8_t *seq,
                                      const int64_t *s1_off, const int32_t *s1_len,
                                      const int64_t *s2_off, const int32_t *s2_len,
                                      const int64_t *m_off, const int32_t *m_len,
                                      const int64_t *p_off, const int32_t *p_len,
                                      int32_t *cost, uint8_t *out, const int64_t *out_off,
                                      int32_t *out_len, int32_t *changed, void *stream) {
  if (!cm) return fail(POYD_EINVAL, "poyd_readjust_3d_batch: null cost matrix");
  if (!cm->combinations || cm->lcm != 5 || cm->gap != 16)
    return fail(POYD_EUNSUP, "poyd_readjust_3d_batch: the DNA alphabet with combinations");
  // align_3_powell_inter's parameters (sequence.ml:1091-1102)
  const int mm = cm->cost[(1 << 5) + 2], ge = cm->cost[(1 << 5) + 16];
  const int go = cm->cost_model == 1 ? cm->gap_open : 0;
  const int64_t *off[4] = {s1_off, s2_off, p_off, m_off};
  const int32_t *len[4] = {s1_len, s2_len, p_len, m_len};
  return p3_run(1, n, seq, off, len, mm, go, ge, cm->gap, nullptr, cm, cost, out, out_off, out_len,
                changed, (cudaStream_t)stream);
}

extern "C" int poyd_powell_3D_align(const uint8_t *sa, int32_t la, const uint8_t *sb,
                                    int32_t lb, const uint8_t *sc, int32_t lc, uint8_t *ra,
                                    uint8_t *rb, uint8_t *rc, int32_t cap, int32_t *len,
                                    int32_t mm, int32_t go, int32_t ge, int32_t *cost) {
  if (!sa || !sb || !sc || !ra || !rb || !rc || !len || !cost)
    return fail(POYD_EINVAL, "poyd_powell_3D_align: null argument");
  if (la < 1 || lb < 1 || lc < 1) return fail(POYD_EINVAL, "poyd_powell_3D_align: empty sequence");
  if ((int64_t)cap < (int64_t)la + lb + lc - 2)
    return fail(POYD_ERANGE, "output capacity below len(a) + len(b) + len(c) - 2");
  Workspace *w = workspace();
  cudaStream_t st = nullptr;
  // staging: [offsets x4 | lengths x3, cost, out_len x2 | a b c | slot]
  const int64_t slot = ((int64_t)la + lb + lc + 3) & ~(int64_t)3;
  const size_t in = ((size_t)la + lb + lc + 63) & ~(size_t)63;
  uint8_t *buf = (uint8_t *)ws_buffer(w, WS_P3_IO, 64 + in + 4 * (size_t)slot);
  if (!buf) return fail(POYD_ENOMEM, "poyd_powell_3D_align: staging allocation failed");
  int64_t *meta = (int64_t *)buf;
  int32_t *m32 = (int32_t *)(buf + 32);
  uint8_t *sq = buf + 64, *o = buf + 64 + in;
  const int64_t hmeta[4] = {0, la, (int64_t)la + lb, 0};
  const int32_t hlen[3] = {la, lb, lc};
  CK3(cudaMemcpyAsync(sq, sa, la, cudaMemcpyHostToDevice, st));
  CK3(cudaMemcpyAsync(sq + la, sb, lb, cudaMemcpyHostToDevice, st));
  CK3(cudaMemcpyAsync(sq + la + lb, sc, lc, cudaMemcpyHostToDevice, st));
  CK3(cudaMemcpyAsync(meta, hmeta, sizeof(hmeta), cudaMemcpyHostToDevice, st));
  CK3(cudaMemcpyAsync(m32, hlen, sizeof(hlen), cudaMemcpyHostToDevice, st));
  int rc_ = poyd_powell_3d_batch(1, sq, meta, m32, meta + 1, m32 + 1, meta + 2, m32 + 2, mm, go,
                                 ge, nullptr, m32 + 3, o, meta + 3, m32 + 4, st);
  if (rc_) return rc_;
  int32_t res[3];
  CK3(cudaMemcpy(res, m32 + 3, sizeof(res), cudaMemcpyDeviceToHost));
  const int n = res[1];
  if (n > cap) return fail(POYD_ERANGE, "poyd_powell_3D_align: alignment longer than cap");
  uint8_t *dst[3] = {ra, rb, rc};
  for (int k = 0; k < 3; ++k)
    CK3(cudaMemcpy(dst[k] + cap - n, o + (k + 1) * slot - n, (size_t)n, cudaMemcpyDeviceToHost));
  *len = n;
  *cost = res[0];
  return POYD_OK;
}
