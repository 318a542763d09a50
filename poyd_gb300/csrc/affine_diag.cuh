// Shared by affine.cu and affine_diag.cu: per-pair plans of the affine path.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "poyd_internal.h"

namespace poyd {

struct AffPlan {
  int64_t si_off, sj_off;
  int32_t leni, lenj;  // rows 0..leni (si), columns 0..lenj (sj)
  int32_t e0, wd;
  int32_t swap;        // 1: rows are the caller's b
  int32_t nstrips, sblocks;  // sblocks: 4-step DM words per lane per strip
  int32_t empty;
  int32_t pad_[4];
};
static_assert(sizeof(AffPlan) == 64, "AffPlan layout");

// Where k_aff_diag left a pair's direction codes.
struct AffWhere {
  int64_t off;    // 32-bit word offset of the pair's task
  int32_t lane0;  // first lane of its group
  int32_t width;  // diagonals per lane
};

struct AffDiagArgs {
  int tasks;
  const uint8_t *seq;
  const AffPlan *plans;
  const int32_t *order;    // kDiagTask slots per task (-1: no pair)
  const int64_t *task;     // aff_diag_task of each task, longest first
  const DevTables *tables;
  int go;
  int *counter;
  uint32_t *dm;
  AffWhere *where;
  int32_t *cost;
  unsigned one, m1, k4, k8, k16, k32, k256;  // multipliers the compiler does not know
};

struct AffWalkArgs {
  int n;
  const uint8_t *seq;
  const AffPlan *plans;
  const int32_t *order;  // the pairs to walk
  const AffWhere *where;
  const uint32_t *dm;
  const DevTables *tables;
  uint8_t *out;
  const int64_t *out_off;
  int32_t *out_len;
};

// A task is a warp's pairs: 32 / lanes of them, `lanes` lanes each with `width`
// diagonals (8 x 12 diagonals up to 32 x 16; 8 a lane in small batches with
// directions alone).
constexpr int kDiagTask = 4;
struct AffDiagClass {
  int lanes, width;
};
constexpr AffDiagClass kDiagClasses[] = {{8, 12},  {8, 16},  {16, 8}, {16, 12},
                                         {16, 16}, {32, 12}, {32, 16}};
constexpr int kDiagClassN = 7;
// Smallest class for a band of e0 (kDiagClassN: wider than all).  `spread`: of 16
// lanes at least (the fewer diagonals a lane, the shorter a pair's own time).
inline int aff_diag_class(int e0, bool spread) {
  int best = kDiagClassN, slots = 1 << 30;
  for (int c = 0; c < kDiagClassN; ++c) {
    const int s = kDiagClasses[c].lanes * kDiagClasses[c].width;
    if (spread ? kDiagClasses[c].lanes < 16 : kDiagClasses[c].width < 12) continue;
    if (s >= e0 + 41 && s < slots) best = c, slots = s;
  }
  return best;
}
// Batches with directions are spread up to eight pairs an SM: 200 pairs of
// 100-5,000 bp take 0.81 ms instead of 1.53, 1,300 of 1,000 bp 0.26 instead of 0.34;
// 2,600 of 1,000 bp would take 0.36 instead of 0.32.  Costs alone gain nothing
// (200 pairs of 1,000 bp: 0.21 ms both ways).
constexpr int kDiagSpreadPerSm = 8;
// Task word: direction words' offset, lanes and width; the words of a task
// whose longest pair has leni + lenj = steps.
inline int64_t aff_diag_task(int64_t off, AffDiagClass c) {
  return off | (int64_t)c.lanes << 56 | (int64_t)c.width << 48;
}
inline int64_t aff_diag_words(int width, int64_t steps) { return (steps / 4 + 1) * 16 * width; }
// spread: with directions, of classes chosen as such
int launch_aff_diag(const AffDiagArgs &A, bool bt, bool gaps, bool spread, cudaStream_t st);
int launch_aff_walk(const AffWalkArgs &A, cudaStream_t st);

}  // namespace poyd
