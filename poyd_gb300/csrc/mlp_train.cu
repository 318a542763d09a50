// Backward pass and optimizer step of the join-proposal MLP, in three
// launches: the chain of dZ's, every weight and bias gradient, and Adam over
// all parameters.  At a training batch of a few thousand rows the work is a
// few GFLOP, so what counts is the number of launches and that each one
// covers the SMs; mma.sync keeps the operands in registers and shared
// memory at these sizes (the products take a few microseconds in all).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "poyd_internal.h"

namespace poyd {
namespace {

constexpr int kTIn = 32, kTH1 = 256, kTH2 = 256, kTH3 = 128;
constexpr int kTThreads = 256;
constexpr int kTRows = 32;   // rows of a chain block
constexpr int kTPad = 8;     // elements after a staged row: conflict-free fragments

struct MlpBwdArgs {
  int M;
  const __nv_bfloat16 *X, *H[3], *W2, *W3, *w4;  // H1, H2, H3; W [in][out]
  const float *y, *target;
  __nv_bfloat16 *dZ[3];                           // dZ1, dZ2, dZ3
  float *gW[4], *gb[4], *loss;
};

__device__ __forceinline__ void t_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                      uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void t_ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ float t_dy(const MlpBwdArgs &A, int m) {
  return 2.f * (A.y[m] - A.target[m]) / (float)A.M;
}

// dZ of a 256-wide layer for the block's 32 rows: (in [32][K] of shared
// memory) . W^T with W [256][K] (so that a B fragment is one 32-bit load from
// L2), masked by the layer's activations.  A warp takes 32 columns; the k
// chunks of 16 are summed in ascending order.
template <int K>
__device__ __forceinline__ void t_chain(const __nv_bfloat16 *in, const __nv_bfloat16 *__restrict__ W,
                                        const __nv_bfloat16 *__restrict__ H, __nv_bfloat16 *dZ,
                                        __nv_bfloat16 *out, int m0, int M, int warp, int lane) {
  constexpr int LD = K + kTPad, LO = 256 + kTPad;
  const int g = lane >> 2, t = lane & 3;
  float acc[2][4][4] = {};
#pragma unroll 8
  for (int k0 = 0; k0 < K; k0 += 16) {
    uint32_t a[2][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      const __nv_bfloat16 *r0 = in + (mt * 16 + g) * LD + k0 + 2 * t;
      a[mt][0] = *reinterpret_cast<const uint32_t *>(r0);
      a[mt][1] = *reinterpret_cast<const uint32_t *>(r0 + 8 * LD);
      a[mt][2] = *reinterpret_cast<const uint32_t *>(r0 + 8);
      a[mt][3] = *reinterpret_cast<const uint32_t *>(r0 + 8 * LD + 8);
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const __nv_bfloat16 *w = W + (int64_t)(warp * 32 + nt * 8 + g) * K + k0 + 2 * t;
      const uint32_t b0 = *reinterpret_cast<const uint32_t *>(w);
      const uint32_t b1 = *reinterpret_cast<const uint32_t *>(w + 8);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) t_mma(acc[mt][nt], a[mt], b0, b1);
    }
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = mt * 16 + g + 8 * q, n = warp * 32 + nt * 8 + 2 * t, m = m0 + r;
        __nv_bfloat162 v = __floats2bfloat162_rn(0.f, 0.f);
        if (m < M) {
          const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(H + (int64_t)m * 256 + n);
          if (__bfloat162float(h.x) > 0.f) v.x = __float2bfloat16_rn(acc[mt][nt][2 * q]);
          if (__bfloat162float(h.y) > 0.f) v.y = __float2bfloat16_rn(acc[mt][nt][2 * q + 1]);
          *reinterpret_cast<__nv_bfloat162 *>(dZ + (int64_t)m * 256 + n) = v;
        }
        if (out) *reinterpret_cast<__nv_bfloat162 *>(out + r * LO + n) = v;
      }
}

// The output bias's gradient and the loss, summed row after row as
// poyd_mlp_head_backward sums them: the residuals cancel, so that another order's
// rounding would show in the sixth digit of the one number.  Two threads add what
// the others have staged, 1,024 rows a turn, by a block of its own beside the chain
// (4,096 rows: 9 of the launch's 22 us).
__device__ __forceinline__ void t_head_sums(const MlpBwdArgs &A, float *buf) {
  constexpr int kTurn = 1024;
  const int tid = threadIdx.x;
  auto stage = [&](int m0, int first, int step) {
    float *d = buf + (m0 / kTurn & 1) * 2 * kTurn, *e = d + kTurn;
    for (int x = first; x < kTurn; x += step) {
      const int m = m0 + x;
      const float r = m < A.M ? A.y[m] - A.target[m] : 0.f;
      e[x] = r;
      d[x] = 2.f * r / (float)A.M;
    }
  };
  stage(0, tid, kTThreads);
  __syncthreads();
  float s = 0.f;
  for (int m0 = 0; m0 < A.M; m0 += kTurn) {
    const float4 *v = reinterpret_cast<const float4 *>(buf + ((m0 / kTurn & 1) * 2 + tid / 32) * kTurn);
    if (tid >= 64) {
      if (m0 + kTurn < A.M) stage(m0 + kTurn, tid - 64, kTThreads - 64);
    } else if (tid == 0) {
#pragma unroll 8
      for (int x = 0; x < kTurn / 4; ++x) {
        const float4 f = v[x];
        s += f.x;
        s += f.y;
        s += f.z;
        s += f.w;
      }
    } else if (tid == 32) {
#pragma unroll 8
      for (int x = 0; x < kTurn / 4; ++x) {
        const float4 f = v[x];
        s = fmaf(f.x, f.x, s);
        s = fmaf(f.y, f.y, s);
        s = fmaf(f.z, f.z, s);
        s = fmaf(f.w, f.w, s);
      }
    }
    __syncthreads();
  }
  if (tid == 0) A.gb[3][0] = s;
  if (tid == 32) A.loss[0] = s / (float)A.M;
}

// dZ3 = dy w4 masked, dZ2 = dZ3 W3^T masked, dZ1 = dZ2 W2^T masked, for 32
// rows a block, whose activations are in shared memory and whose weights come from
// L2; the first block takes t_head_sums.
__global__ void __launch_bounds__(kTThreads) k_mlp_chain(const __grid_constant__ MlpBwdArgs A) {
  __shared__ __align__(16) __nv_bfloat16 z3[kTRows * (kTH3 + kTPad)];
  __shared__ __align__(16) __nv_bfloat16 z2[kTRows * (kTH2 + kTPad)];
  static_assert(sizeof(z2) >= 4 * 1024 * sizeof(float), "t_head_sums stages over z2");
  if (blockIdx.x == 0) {
    t_head_sums(A, reinterpret_cast<float *>(z2));
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = (blockIdx.x - 1) * kTRows;
  __shared__ float dy[kTRows];
  if (threadIdx.x < kTRows) {
    const int m = m0 + threadIdx.x;
    dy[threadIdx.x] = m < A.M ? t_dy(A, m) : 0.f;
  }
  // eight columns a thread, two rows
  const int c8 = (threadIdx.x & 15) * 8;
  uint4 h4[2];
  float w[8];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int m = m0 + (threadIdx.x >> 4) + 16 * q;
    h4[q] = m < A.M ? *reinterpret_cast<const uint4 *>(A.H[2] + (int64_t)m * kTH3 + c8)
                    : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = __bfloat162float(A.w4[c8 + i]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int r = (threadIdx.x >> 4) + 16 * q, m = m0 + r;
    const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&h4[q]);
    uint4 o;
    __nv_bfloat16 *v = reinterpret_cast<__nv_bfloat16 *>(&o);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = __float2bfloat16_rn(__bfloat162float(h[i]) > 0.f ? dy[r] * w[i] : 0.f);
    if (m < A.M) *reinterpret_cast<uint4 *>(A.dZ[2] + (int64_t)m * kTH3 + c8) = o;
    *reinterpret_cast<uint4 *>(z3 + r * (kTH3 + kTPad) + c8) = o;
  }
  __syncthreads();
  t_chain<kTH3>(z3, A.W3, A.H[1], A.dZ[1], z2, m0, A.M, warp, lane);
  __syncthreads();
  t_chain<kTH2>(z2, A.W2, A.H[0], A.dZ[0], nullptr, m0, A.M, warp, lane);
}

// Gradients: dW = a_in^T dZ is a reduction over the batch, so a 64 x 128 tile
// of a gradient is shared by a cluster of 8 blocks, each with an eighth of
// the rows; the partial tiles meet in distributed shared memory and are
// summed in rank order (the same sum every time).  Tiles 0-1: layer 1 (its 32
// rows fill half a tile), 2-9: layer 2, 10-13: layer 3; the tile with input
// row 0 also sums dZ's columns (the bias gradient).  Tile 14: the head's dw.
// Measured at 4,096 rows against one reduction over the
// whole batch per tile: 8-64 blocks were busy for most of 1.5 ms.
constexpr int kGSplit = 8, kGTiles = 15;
constexpr int kGM = 64, kGN = 128, kGK = 32;  // tile and staged rows
constexpr int kGLdA = kGM + kTPad, kGLdB = kGN + kTPad;
static_assert(4 * kGK * (kGLdA + kGLdB) <= 4 * (kGM + 1) * kGN, "two stages fit under the tile");

__global__ void __cluster_dims__(kGSplit, 1, 1) __launch_bounds__(kTThreads)
    k_mlp_grads(const __grid_constant__ MlpBwdArgs A) {
  namespace cg = cooperative_groups;
  // the staged rows, then (over them) the partial tile and its column sums
  __shared__ __align__(16) float part[(kGM + 1) * kGN];
  __nv_bfloat16 *const stage = reinterpret_cast<__nv_bfloat16 *>(part);
  auto sa = [&](int s) { return stage + s * kGK * kGLdA; };
  auto sb = [&](int s) { return stage + 2 * kGK * kGLdA + s * kGK * kGLdB; };
  auto cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tile = blockIdx.x / kGSplit;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this rank's rows, whole 16-row chunks
  const int chunk = ((A.M + kGSplit - 1) / kGSplit + 15) & ~15;
  const int r0 = min(A.M, rank * chunk), r1 = min(A.M, r0 + chunk);
  int rows = kGM;  // gradient rows of the tile
  if (tile == kGTiles - 1) {
    // [0, 128): dw.  256 rows a pass: their dy into shared memory, then eight
    // columns a thread over every 16th row.
    float *dyv = part + 16 * 128;
    const int c8 = (tid & 15) * 8, rg = tid >> 4;
    float sw[8] = {};
    for (int m = r0; m < r1; m += kTThreads) {
      const float d = m + tid < r1 ? t_dy(A, m + tid) : 0.f;
      __syncthreads();
      dyv[tid] = d;
      __syncthreads();
#pragma unroll 8
      for (int i = 0; i < kTThreads / 16; ++i) {
        const int r = rg + 16 * i;
        uint4 h4 = make_uint4(0, 0, 0, 0);
        if (m + r < r1)
          h4 = __ldg(reinterpret_cast<const uint4 *>(A.H[2] + (int64_t)(m + r) * kTH3 + c8));
        const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&h4);
#pragma unroll
        for (int j = 0; j < 8; ++j) sw[j] = fmaf(__bfloat162float(h[j]), dyv[r], sw[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) part[rg * 128 + c8 + j] = sw[j];
    __syncthreads();
    float t = 0.f;
    if (tid < 128)
      for (int g = 0; g < 16; ++g) t += part[g * 128 + tid];
    __syncthreads();
    if (tid < 128) part[tid] = t;
  } else {
    const int layer = tile < 2 ? 0 : tile < 10 ? 1 : 2;
    const int lt = tile - (layer == 0 ? 0 : layer == 1 ? 2 : 10);
    const int K = layer == 0 ? kTIn : 256, N = layer == 2 ? kTH3 : 256;
    const int ib = (N == 256 ? lt >> 1 : lt) * kGM, nb = N == 256 ? (lt & 1) * kGN : 0;
    const __nv_bfloat16 *in = layer == 0 ? A.X : A.H[layer - 1], *dz = A.dZ[layer];
    rows = min(kGM, K - ib);
    // a staged row: 64 input columns (8 threads) and 128 dZ columns (16)
    const int ar = tid >> 3, ac = tid & 7, br = tid >> 4, bc = tid & 15;
    const bool acol = ib + 8 * ac < K;
    uint4 va, vb[2];
    auto fetch = [&](int m) {
      va = vb[0] = vb[1] = make_uint4(0, 0, 0, 0);
      if (acol && m + ar < r1)
        va = *reinterpret_cast<const uint4 *>(in + (int64_t)(m + ar) * K + ib + 8 * ac);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (m + br + 16 * q < r1)
          vb[q] = *reinterpret_cast<const uint4 *>(dz + (int64_t)(m + br + 16 * q) * N + nb + 8 * bc);
    };
    auto put = [&](int s) {
      *reinterpret_cast<uint4 *>(&sa(s)[ar * kGLdA + 8 * ac]) = va;
#pragma unroll
      for (int q = 0; q < 2; ++q)
        *reinterpret_cast<uint4 *>(&sb(s)[(br + 16 * q) * kGLdB + 8 * bc]) = vb[q];
    };
    const int wm = warp & 1, wn = warp >> 1;  // 32 x 32 of the tile
    float acc[2][4][4] = {};
    float bsum = 0.f;
    const int bcol = tid & 127, bhalf = tid >> 7;
    fetch(r0);
    put(0);
    __syncthreads();
    int s = 0;
    for (int m = r0; m < r1; m += kGK, s ^= 1) {
      if (m + kGK < r1) fetch(m + kGK);
      if (ib == 0) {
#pragma unroll
        for (int r = 0; r < kGK / 2; ++r)
          bsum += __bfloat162float(sb(s)[(2 * r + bhalf) * kGLdB + bcol]);
      }
      const uint32_t pa = (uint32_t)__cvta_generic_to_shared(sa(s));
      const uint32_t pb = (uint32_t)__cvta_generic_to_shared(sb(s));
#pragma unroll
      for (int k0 = 0; k0 < kGK; k0 += 16) {
        // transposed 8x8 loads: A's four are (m, k), (m + 8, k), (m, k + 8),
        // (m + 8, k + 8); B's (k, n), (k + 8, n), (k, n + 8), (k + 8, n + 8)
        uint32_t a[2][4], b[2][4];
        const int q = lane >> 3, l8 = lane & 7;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          t_ldsm4t(a[i], pa + 2 * ((k0 + l8 + 8 * (q >> 1)) * kGLdA + wm * 32 + i * 16 + 8 * (q & 1)));
          t_ldsm4t(b[i], pb + 2 * ((k0 + l8 + 8 * (q & 1)) * kGLdB + wn * 32 + i * 16 + 8 * (q >> 1)));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) t_mma(acc[i][j], a[i], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
      }
      if (m + kGK < r1) put(s ^ 1);
      __syncthreads();
    }
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          part[(wm * 32 + i * 16 + g + (q >> 1) * 8) * kGN + wn * 32 + j * 8 + 2 * t + (q & 1)] = acc[i][j][q];
    if (bhalf) part[kGM * kGN + bcol] = bsum;
    __syncthreads();
    if (!bhalf) part[kGM * kGN + bcol] += bsum;
  }
  cluster.sync();
  // each rank sums an eighth of the tile's rows over the ranks
  const float *peer[kGSplit];
#pragma unroll
  for (int r = 0; r < kGSplit; ++r) peer[r] = cluster.map_shared_rank(part, r);
  auto total = [&](int i) {
    float s = peer[0][i];
#pragma unroll
    for (int r = 1; r < kGSplit; ++r) s += peer[r][i];
    return s;
  };
  if (tile == kGTiles - 1) {
    if (rank == 0 && tid < 128) A.gW[3][tid] = total(tid);
  } else {
    const int layer = tile < 2 ? 0 : tile < 10 ? 1 : 2;
    const int lt = tile - (layer == 0 ? 0 : layer == 1 ? 2 : 10);
    const int N = layer == 2 ? kTH3 : 256;
    const int ib = (N == 256 ? lt >> 1 : lt) * kGM, nb = N == 256 ? (lt & 1) * kGN : 0;
    for (int e = tid; e < kGM / kGSplit * kGN; e += kTThreads) {
      const int r = rank * (kGM / kGSplit) + e / kGN, c = e % kGN;
      if (r < rows) A.gW[layer][(int64_t)(ib + r) * N + nb + c] = total(r * kGN + c);
    }
    if (ib == 0 && rank == kGSplit - 1 && tid < kGN) A.gb[layer][nb + tid] = total(kGM * kGN + tid);
  }
  cluster.sync();  // the peers have read this block's part
}

// Adam on fp32 master weights, refreshing the bf16 copies: several tensors a
// launch.
constexpr int kAdamMost = 16;
struct AdamArgs {
  int n;
  int64_t end[kAdamMost];  // running element counts
  float *w[kAdamMost], *m[kAdamMost], *v[kAdamMost];
  const float *g[kAdamMost];
  __nv_bfloat16 *w16[kAdamMost];
  float lr, b1, b2, eps, c1, c2;
};
__global__ void k_adam_all(const __grid_constant__ AdamArgs A) {
  const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int t = 0;
  while (t < A.n && x >= A.end[t]) ++t;
  if (t == A.n) return;
  const int64_t i = x - (t ? A.end[t - 1] : 0);
  const float gi = A.g[t][i];
  const float m = A.b1 * A.m[t][i] + (1.f - A.b1) * gi;
  const float v = A.b2 * A.v[t][i] + (1.f - A.b2) * gi * gi;
  A.m[t][i] = m;
  A.v[t][i] = v;
  const float w = A.w[t][i] - A.lr * (m / A.c1) / (sqrtf(v / A.c2) + A.eps);
  A.w[t][i] = w;
  if (A.w16[t]) A.w16[t][i] = __float2bfloat16_rn(w);
}

}  // namespace
}  // namespace poyd

using namespace poyd;

extern "C" int poyd_mlp_backward(const void *X, int32_t M, const void *H1, const void *H2,
                                 const void *H3, const void *W2, const void *W3, const void *w4,
                                 const float *y, const float *target, void *dZ, float *const *gW,
                                 float *const *gb, float *loss, void *stream) {
  if (M < 1 || !X || !H1 || !H2 || !H3 || !W2 || !W3 || !w4 || !y || !target || !dZ || !gW || !gb ||
      !loss)
    return fail(POYD_EINVAL, "poyd_mlp_backward: bad arguments");
  for (const void *p : {X, H1, H2, H3, (const void *)dZ})
    if ((uintptr_t)p & 15) return fail(POYD_EINVAL, "poyd_mlp_backward: rows must be 16-byte aligned");
  if (((uintptr_t)W2 | (uintptr_t)W3) & 3)
    return fail(POYD_EINVAL, "poyd_mlp_backward: weights must be 4-byte aligned");
  MlpBwdArgs A = {};
  A.M = M;
  A.X = (const __nv_bfloat16 *)X;
  const void *H[3] = {H1, H2, H3};
  for (int i = 0; i < 3; ++i) A.H[i] = (const __nv_bfloat16 *)H[i];
  A.W2 = (const __nv_bfloat16 *)W2;
  A.W3 = (const __nv_bfloat16 *)W3;
  A.w4 = (const __nv_bfloat16 *)w4;
  A.y = y;
  A.target = target;
  A.dZ[0] = (__nv_bfloat16 *)dZ;
  A.dZ[1] = A.dZ[0] + (int64_t)M * kTH1;
  A.dZ[2] = A.dZ[1] + (int64_t)M * kTH2;
  for (int i = 0; i < 4; ++i) {
    if (!gW[i] || !gb[i]) return fail(POYD_EINVAL, "poyd_mlp_backward: null gradient");
    A.gW[i] = gW[i];
    A.gb[i] = gb[i];
  }
  A.loss = loss;
  cudaStream_t st = (cudaStream_t)stream;
  {
    ProfScope ps("mlp_chain", st);
    k_mlp_chain<<<(M + kTRows - 1) / kTRows + 1, kTThreads, 0, st>>>(A);
  }
  {
    ProfScope ps("mlp_grads", st);
    k_mlp_grads<<<kGTiles * kGSplit, kTThreads, 0, st>>>(A);
  }
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "poyd_mlp_backward") : POYD_OK;
}

extern "C" int poyd_adam_step_all(int32_t n, float *const *w, void *const *w16,
                                  const float *const *g, float *const *m, float *const *v,
                                  const int64_t *sizes, float lr, float b1, float b2, float eps,
                                  int32_t step, void *stream) {
  if (n < 0 || n > kAdamMost || (n && (!w || !w16 || !g || !m || !v || !sizes)))
    return fail(POYD_EINVAL, "poyd_adam_step_all: bad arguments (at most %d tensors)", kAdamMost);
  AdamArgs A = {};
  A.n = n;
  int64_t total = 0;
  for (int i = 0; i < n; ++i) {
    if (sizes[i] < 0 || (sizes[i] && (!w[i] || !g[i] || !m[i] || !v[i])))
      return fail(POYD_EINVAL, "poyd_adam_step_all: tensor %d", i);
    total += sizes[i];
    A.end[i] = total;
    A.w[i] = w[i];
    A.w16[i] = (__nv_bfloat16 *)w16[i];
    A.g[i] = g[i];
    A.m[i] = m[i];
    A.v[i] = v[i];
  }
  if (total == 0) return POYD_OK;
  A.lr = lr;
  A.b1 = b1;
  A.b2 = b2;
  A.eps = eps;
  A.c1 = 1.f - powf(b1, (float)step);
  A.c2 = 1.f - powf(b2, (float)step);
  cudaStream_t st = (cudaStream_t)stream;
  {
    ProfScope ps("mlp_adam", st);
    k_adam_all<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(A);
  }
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? cuda_fail(e, "poyd_adam_step_all") : POYD_OK;
}

extern "C" int poyd_adam_step(float *w, void *w16, const float *g, float *m, float *v, int64_t n,
                              float lr, float b1, float b2, float eps, int32_t step,
                              void *stream) {
  if (n <= 0) return POYD_OK;
  return poyd_adam_step_all(1, &w, &w16, &g, &m, &v, &n, lr, b1, b2, eps, step, stream);
}
