// Layouts of batched results: output slots sized by the inputs' lengths, and the
// places of packed results.  One launch and one read-back each (the running sum
// of a few tensor operations took a dozen launches and two waits, 100-150 us of
// a call on one pair).  No reference counterpart: the reference hands back one
// seq block per call.
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>
#include "poyd_internal.h"
#include "linear_kernels.cuh"

namespace poyd {
namespace {

constexpr int kLayThreads = 1024, kLayItems = 8;

struct LayoutArgs {
  int n;
  const int32_t *l0, *l1, *l2;  // slots: the lengths (l2 may be null)
  int extra;                    // ... and the bytes on top of them
  const int32_t *out_len;       // packed results: lengths of the alignments
  int64_t *off, *cap;
  int64_t *total;               // bytes in all; the least out_len
};

// Exclusive running sum by one block, eight items a thread: the batch's lengths
// are read once, 1.6 MB at 200,000 pairs.  Bound: the latency of a round, 10 us each
// (align.py sizes more than 65,536 pairs by tensor operations).
template <bool PACK>
__global__ void __launch_bounds__(kLayThreads) k_layout(const LayoutArgs A) {
  __shared__ int64_t part[32];
  __shared__ int64_t s_run;
  __shared__ int low[32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int64_t run = 0;
  int least = INT32_MAX;
  for (int64_t base = 0; base < A.n; base += kLayThreads * kLayItems) {
    int64_t v[kLayItems], sum = 0;
#pragma unroll
    for (int e = 0; e < kLayItems; ++e) {
      const int64_t i = base + (int64_t)t * kLayItems + e;
      v[e] = 0;
      if (i < A.n) {
        if (PACK) {
          const int a = A.out_len[2 * i], m = A.out_len[2 * i + 1];
          least = min(least, min(a, m));
          v[e] = 3 * (int64_t)a + m;
        } else {
          const int64_t c = ((int64_t)A.l0[i] + A.l1[i] + (A.l2 ? A.l2[i] : 0) + A.extra + 3) & ~(int64_t)3;
          A.cap[i] = c;
          v[e] = 4 * c;
        }
      }
      sum += v[e];
    }
    int64_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int64_t x = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += x;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int64_t p = part[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int64_t x = __shfl_up_sync(0xffffffffu, p, d);
        if (lane >= d) p += x;
      }
      part[lane] = p;
    }
    __syncthreads();
    int64_t at = run + (warp ? part[warp - 1] : 0) + incl - sum;
#pragma unroll
    for (int e = 0; e < kLayItems; ++e) {
      const int64_t i = base + (int64_t)t * kLayItems + e;
      if (i < A.n) A.off[i] = at;
      at += v[e];
    }
    if (t == kLayThreads - 1) s_run = at;
    __syncthreads();
    run = s_run;
  }
  if (PACK) {
    least = __reduce_min_sync(0xffffffffu, least);
    if (lane == 0) low[warp] = least;
    __syncthreads();
    if (warp == 0) least = __reduce_min_sync(0xffffffffu, low[lane]);
  }
  if (t == 0) {
    A.total[0] = run;
    A.total[1] = least;
  }
}

// Unlike other calls, layouts of several threads may overlap on a stream: a caller
// whose batches have streams of their own sizes them on the current one.
int layout(const LayoutArgs &in, bool pack, int64_t *total, int64_t *least, cudaStream_t st) {
  LayoutArgs A = in;
  Workspace *w = workspace(st);
  std::lock_guard<std::mutex> lk(ws_layout_mutex(w));
  A.total = (int64_t *)ws_buffer(w, WS_LAYOUT, 2 * sizeof(int64_t));
  if (!A.total) return fail(POYD_ENOMEM, "layout allocation failed");
  if (pack) k_layout<true><<<1, kLayThreads, 0, st>>>(A);
  else k_layout<false><<<1, kLayThreads, 0, st>>>(A);
  int64_t h[2];
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, A.total, sizeof h, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "result layout");
  *total = h[0];
  if (least) *least = h[1];
  return POYD_OK;
}

}  // namespace
}  // namespace poyd

using namespace poyd;

extern "C" int poyd_slot_layout(int32_t n, const int32_t *len0, const int32_t *len1,
                                const int32_t *len2, int32_t extra, int64_t *out_off, int64_t *cap,
                                int64_t *total, void *stream) {
  if (n < 0 || !total || (n > 0 && (!len0 || !len1 || !out_off || !cap)))
    return fail(POYD_EINVAL, "poyd_slot_layout: null argument");
  *total = 0;
  if (n == 0) return POYD_OK;
  LayoutArgs A = {};
  A.n = n; A.l0 = len0; A.l1 = len1; A.l2 = len2; A.extra = extra; A.off = out_off; A.cap = cap;
  return layout(A, false, total, nullptr, (cudaStream_t)stream);
}

extern "C" int poyd_pack_layout(int32_t n, const int32_t *out_len, int64_t *packed_off,
                                int64_t *total, int64_t *least, void *stream) {
  if (n < 0 || !total || !least || (n > 0 && (!out_len || !packed_off)))
    return fail(POYD_EINVAL, "poyd_pack_layout: null argument");
  *total = *least = 0;
  if (n == 0) return POYD_OK;
  LayoutArgs A = {};
  A.n = n; A.out_len = out_len; A.off = packed_off;
  return layout(A, true, total, least, (cudaStream_t)stream);
}

extern "C" int poyd_pack_slots(int32_t n, const uint8_t *out, const int64_t *out_off,
                               const int64_t *cap, const int32_t *out_len, uint8_t *packed,
                               const int64_t *packed_off, void *stream) {
  if (n < 0 || (n > 0 && (!out || !out_off || !cap || !out_len || !packed || !packed_off)))
    return fail(POYD_EINVAL, "poyd_pack_slots: null argument");
  if (n == 0) return POYD_OK;
  cudaStream_t st = (cudaStream_t)stream;
  {
    ProfScope ps("pack_alignments", st);
    launch_pack_alignments(n, out, out_off, nullptr, nullptr, cap, out_len, packed, packed_off, st);
  }
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "poyd_pack_slots") : POYD_OK;
}
