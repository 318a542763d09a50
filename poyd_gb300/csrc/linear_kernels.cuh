// Argument blocks and launchers of the linear-gap kernels (linear.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "poyd_internal.h"

namespace poyd {

struct LinPlanArgs {
  int n;
  const uint8_t *seq;
  const int64_t *a_off;
  const int32_t *a_len;
  const int64_t *b_off;
  const int32_t *b_len;
  int policy;
  const int32_t *deltaw;
  int gap;
  int maxc;
  int with_dm;  // kDpCost, kDpSets or kDpChoice: sizes the direction matrix
  int dos_empty;
  LinPlan *plans;
  int64_t *dm_words;
  int32_t *wd_out;
  int64_t *cells;
  int32_t *err;
};

struct LinTbArgs {
  int n;
  const uint8_t *seq;
  const LinPlan *plans;
  const int64_t *dm_off;
  const uint32_t *dm;
  const DevTables *tables;
  int gap;
  uint8_t *out;
  const int64_t *out_off;
  int32_t *out_len;
  int swaped;  // -1: derive from the orientation, else backtrack_2d's flag
  int mode;    // kDpSets or kDpChoice: how the direction matrix was written
  const int32_t *order;  // k_lin_traceback: thread t walks pair order[t] (nullable)
};

// Runtime multipliers of the DP's multiply-add arithmetic (see linear.cu).
struct DpK {
  int one, m1, four, m64k, k64;
};
inline DpK dp_constants() { return DpK{1, -1, 4, -65536, 65536}; }

struct LinDpArgs {
  int n;
  const uint8_t *seq;
  const LinPlan *plans;
  const int64_t *dm_off;
  const int32_t *order;
  const DevTables *tables;
  int gap;
  int *counter;
  int *scratch;   // per-warp boundary-row slabs
  int64_t slab;   // ints per slab
  uint32_t *dm;
  int32_t *cost;
  int swaped;  // kDpChoice priority: -1 derives it from the orientation
  // kDpChoice with fuse_tb: the warp finishing the last DP of 32 consecutive
  // pairs (order positions 32b..32b+31, counted in batch_done[b]) runs their
  // traceback with `tb`
  int fuse_tb;
  int *batch_done;
  // with fuse_tb: done[b] = 1 once batch b's results are written (host-mapped
  // memory a caller polls to download finished slots early; may be null)
  int *done;
  // with fuse_tb, packed kernel: every pair has its own warp (n <= warps of
  // the grid) and no done flags are kept, so the warp that filled a pair
  // walks it at once, all lanes together (latency of small batches)
  int tb_solo;
  LinTbArgs tb;
  DpK k;  // multiplier constants (1, -1, 4, -65536)
};

// Device-side pair order and direction-matrix offsets (one launch wave):
// pairs are bucketed by log2 of their lane-steps (32 buckets per octave,
// longest first) and given disjoint direction-matrix regions.
struct LinOrderScratch {
  int hist[1024];           // pairs per bucket, then the scatter cursors
  int base[1024];           // first order position of each bucket
  unsigned long long total; // direction-matrix words of the batch
  int maxwd;                // widest band
  int pad;                  // the plan's error bits
  int maxsum;               // largest l1 + l2 (k_order_small)
  int pad2;
};
void launch_lin_order(int n, const LinPlan *plans, const int64_t *dm_words, int64_t *dm_off,
                      LinOrderScratch *os, int32_t *order, cudaStream_t st);
constexpr int kOrderSmall = 1024;  // batches up to this size use k_order_small
void launch_lin_order_small(int n, const LinPlan *plans, const int64_t *dm_words,
                            int64_t *dm_off, LinOrderScratch *os, int *counter, int *batch_done,
                            int nbatch, cudaStream_t st);

// LinPlanArgs::err: some pair's band does not hold both ends of a path.
constexpr int kPlanNoPath = 32;
void launch_lin_plan(const LinPlanArgs &A, cudaStream_t st);
int lin_dp_blocks(int mode);
void launch_lin_dp(const LinDpArgs &A, int mode, int blocks, cudaStream_t st);
// Packed DP (linear4.cu): four rows per lane in 16-bit halves, kDpCost or
// kDpChoice, for batches the plan marks eligible (no err bit 16).
int lin_dp4_blocks(int mode);
int lin_dp4_warps();
void launch_lin_dp4(const LinDpArgs &A, int mode, int blocks, cudaStream_t st);
// Low-latency DP (linear_team.cu): a block per pair, for small batches that
// k_lin_dp4 could run.  lin_team_width: diagonals per lane for the batch's
// widest band and longest pair (0: does not fit); lin_team_words: direction
// matrix words per pair.
constexpr uint32_t kTeamSmemMax = 200 * 1024;
int lin_team_width(int maxwd, int maxsum);
int64_t lin_team_words(int width, int maxsum);
int launch_lin_team(const LinDpArgs &D, int mode, int width, int64_t dm_stride, int maxsum,
                    cudaStream_t st);
// Throughput DP (linear_diag.cu): 8, 16 or 32 lanes a pair, the band in
// registers, for large batches that k_lin_dp4 could run.  A class is (lanes,
// diagonals a lane), widest band first; wider pairs stay with k_lin_dp4.
struct LinDiagClass {
  int lanes, width;
};
constexpr int kLinDiagClasses = 18, kLinDiagBuckets = 128;
__host__ __device__ __forceinline__ LinDiagClass lin_diag_class(int c) {
  return LinDiagClass{32 >> (c / 6), 28 - 4 * (c % 6)};
}
// idx = j - i + off: the least even off that leaves idx 0 below the band
__host__ __device__ __forceinline__ int lin_diag_off(int dlo) { return (2 - dlo) & ~1; }
// The class of fewest diagonals that holds the band, the fewest lanes among
// equals (kLinDiagClasses: none).
__host__ __device__ __forceinline__ int lin_diag_class_of(int dlo, int wd, int min_lanes) {
  const int need = dlo + lin_diag_off(dlo) + wd;
  int best = kLinDiagClasses, slots = 1 << 30;
  for (int c = 0; c < kLinDiagClasses; ++c) {
    const LinDiagClass k = lin_diag_class(c);
    const int s = k.lanes * k.width;
    if (k.lanes >= min_lanes && s >= need && s <= slots) best = c, slots = s;
  }
  return best;
}
// Double steps whose moves share a direction word: those a lane unrolls.
__host__ __device__ constexpr int lin_diag_block(int width) {
  return width > 12 ? width / 4 : width / 2;
}
// Direction words of a pair of l1 + l2 = sum.
__host__ __device__ __forceinline__ int64_t lin_diag_words(int c, int sum) {
  const LinDiagClass k = lin_diag_class(c);
  return (int64_t)((sum > 2 ? (sum - 2) / 2 : 0) / lin_diag_block(k.width) + 1) * (k.width / 2) * k.lanes;
}
struct LinDiagOrder {
  int hist[(kLinDiagClasses + 1) * kLinDiagBuckets];  // pairs per bucket, then cursors
  // read back in one piece:
  int base[kLinDiagClasses + 1];     // first position of each class; the pairs of none last
  unsigned long long total, total4;  // direction words: this kernel's classes, k_lin_dp4 alone
  int maxwd, err;
  int counter;
};
struct LinDiagArgs {
  int base[kLinDiagClasses + 1], tasks[kLinDiagClasses + 1];
  const uint8_t *seq;
  const LinPlan *plans;
  const int32_t *order;
  const int64_t *dm_off;
  const DevTables *tables;
  int *counter;
  uint32_t *dm;
  int32_t *cost;
  LinTbArgs tb;
  DpK k;
};
int lin_diag_min_lanes(int n, int sms, bool bt);
void launch_lin_diag_order(int n, int min_lanes, bool bt, const LinPlan *plans,
                           const int64_t *dm_words, int64_t *dm_off, LinDiagOrder *os,
                           int32_t *order, cudaStream_t st);
int launch_lin_diag(LinDiagArgs &A, bool bt, const int *base, cudaStream_t st);
int launch_lin_diag_walk(const LinDiagArgs &A, cudaStream_t st);  // after it, the same arguments
// done[b0 .. b1 - 1] = 1 (host-mapped), once what was launched before is written
int launch_lin_diag_flags(int *done, int b0, int b1, cudaStream_t st);
void launch_lin_traceback(const LinTbArgs &A, cudaStream_t st);
void launch_pack_alignments(int n, const uint8_t *out, const int64_t *out_off,
                            const int32_t *a_len, const int32_t *b_len, const int64_t *caps,
                            const int32_t *out_len, uint8_t *packed,
                            const int64_t *packed_off, cudaStream_t st);

}  // namespace poyd
