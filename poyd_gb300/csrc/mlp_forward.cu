// Forward pass of the 32-256-256-128-1 join-proposal MLP, fused into one
// launch on the tcgen05 tensor cores: inference over a pass's candidates and,
// with the activations written out, the training forward.
//
// A CTA keeps all three weight matrices in shared memory (208 KB, staged once)
// and runs 128-row tiles through the layers.  TMEM is two regions of 256 columns,
// P and Q, which change places from tile to tile.  Per tile:
//   * layer 1: A = the tile's bf16 inputs in shared memory, D in P;
//   * the epilogue reads a row's sums with tcgen05.ld (sixteen warps, a thread per
//     row and 32 columns of each half of the layer), adds the bias, applies ReLU, rounds to bf16 and
//     writes the packed values back with tcgen05.st over columns it has read:
//     the next layer's A operand never leaves TMEM, which is what leaves the
//     shared memory to the weights;
//   * layer 2: A from P, D in Q; layer 3: A from Q, D in P's first half.  A
//     layer's products over the first half of its k start when that half of its A
//     is ready and run beside the other half's epilogue;
//   * the 128 -> 1 head from registers by four warps of its own, while the others
//     take the next tile's layer 1, whose sums go to Q.
// Measured: 984,102 rows from fp32 in 0.203 ms (1.03 PFLOP/s; 0.226 where the code
// that keeps activations was not a kernel of its own) where eight warps
// with one tile's products and epilogues in turn took 0.29 ms, and the mma.sync
// kernel with its weights in L2 1.21 ms, the input's conversion and the weights'
// transposes 33 us more.  What bounds it: the chain of a tile, 0.144 ms of it the
// products and the waits around them (0.11 at the tensor cores' rate); a second
// tile's products beside it would want 1,024 TMEM columns.  Layer 2 in halves of
// n, its first half's epilogue beside the second's products, took 0.238 ms.
//
// Every layer accumulates k in ascending chunks of 16 from zero and the head
// sums as k_head_forward does (lane-strided, then the xor butterfly's tree).
//
// B and the layer 1 A operand are K-major without swizzle: 8 x 16-byte core
// matrices, K-adjacent ones 128 bytes apart, 8-row groups 128 * K / 8 + 16
// bytes apart (the 16 bytes spread the staging stores over the banks).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "poyd_internal.h"

namespace poyd {
namespace {

constexpr int kMRows = 128, kMMain = 512, kMThreads = kMMain + 128;
constexpr int kMIn = 32, kMH1 = 256, kMH2 = 256, kMH3 = 128;
__host__ __device__ constexpr int m_sbo(int k) { return k / 8 * 128 + 16; }
constexpr uint32_t kMW1 = 0;
constexpr uint32_t kMW2 = kMW1 + kMH1 / 8 * m_sbo(kMIn);
constexpr uint32_t kMW3 = kMW2 + kMH2 / 8 * m_sbo(kMH1);
constexpr uint32_t kMX = kMW3 + kMH3 / 8 * m_sbo(kMH2);
constexpr uint32_t kMBias = kMX + kMRows / 8 * m_sbo(kMIn);  // b1, b2, b3, w4 (fp32)
constexpr uint32_t kMBar = kMBias + 4 * (kMH1 + kMH2 + 2 * kMH3);
constexpr uint32_t kMSmem = kMBar + 48 + 128;  // + alignment slack
static_assert(kMSmem <= 227 * 1024, "weights, inputs and biases fit one CTA");
constexpr int kMWaitMax = 1 << 20;  // waits of a microsecond before one gives up

struct MlpFwdArgs {
  const void *X;
  int x32;      // X is fp32 (converted here), else bf16
  int trans;    // weights are [out][in] rows, else [in][out]
  int M;
  const uint16_t *W[3];
  const float *b[3];
  const uint16_t *w4;
  const float *b4;
  uint16_t *H[3];  // activations [M][256], [M][256], [M][128], or null
  float *y;
};

__host__ __device__ constexpr int m_tiles(int rows) {
  return (int)(((int64_t)rows + kMRows - 1) / kMRows);
}
__device__ __forceinline__ uint64_t m_desc(uint32_t addr, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(128 >> 4) << 16 |
         (uint64_t)(sbo >> 4) << 32 | 1ull << 46;
}
// kind::f16: fp32 accumulator, bf16 A and B, both K-major
__host__ __device__ constexpr uint32_t m_idesc(int n) {
  return 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(n >> 3) << 17 | (uint32_t)(kMRows >> 4) << 24;
}

__device__ __forceinline__ void m_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void m_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void m_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ bool m_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < kMWaitMax; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(1000)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// The .aligned instructions, the main warps' barrier among them, want the whole
// warp.  Lanes part in waits, in what one thread does alone and in loads of rows
// past M: a __syncwarp() follows each of these (0.8 % of 984,102 rows' time; one
// before every such instruction 1.5 %).  Activations are stored by predicate.
__device__ __forceinline__ void m_ld32(uint32_t (&r)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void m_st16(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 16 bytes at p unless it is null, without a branch.
__device__ __forceinline__ void m_keep(void *p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u64 p, %0, 0;\n@p st.global.v4.b32 [%0], {%1, %2, %3, %4};\n}\n" ::"l"(p),
      "r"(a), "r"(b), "r"(c), "r"(d)
      : "memory");
}
__device__ __forceinline__ void m_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void m_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ uint32_t m_relu2(float lo, float hi) {  // NaN becomes 0
  lo = fmaxf(lo, 0.f);
  hi = fmaxf(hi, 0.f);
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
// {a, b} + {x, y}, ReLU, bf16
__device__ __forceinline__ uint32_t m_bias_relu(uint32_t a, uint32_t b, float x, float y) {
  float lo, hi;
  asm("{\n.reg .b64 s, t;\nmov.b64 s, {%2, %3};\nmov.b64 t, {%4, %5};\nadd.rn.f32x2 s, s, t;\n"
      "mov.b64 {%0, %1}, s;\n}\n"
      : "=f"(lo), "=f"(hi)
      : "r"(a), "r"(b), "f"(x), "f"(y));
  return m_relu2(lo, hi);
}
// Barrier of the sixteen warps of the hidden layers; whether any of them saw `bad`
// (the same answer for all).
__device__ __forceinline__ bool m_main_sync(int bad) {
  int any;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\n"
      "selp.s32 %0, 1, 0, q;\n}\n"
      : "=r"(any)
      : "r"(bad), "n"(kMMain)
      : "memory");
  return any != 0;
}

// Stages a K x N weight matrix as the K-major B operand at `dst`.
__device__ __forceinline__ void m_stage_w(uint8_t *dst, const uint16_t *W, int K, int N,
                                          int trans) {
  const int sbo = m_sbo(K);
  const bool al = ((uintptr_t)W & 15) == 0;
  if (trans) {  // [n][k]: a core matrix row is 16 contiguous bytes
    for (int e = threadIdx.x; e < N * (K / 8); e += kMThreads) {
      const int n = (e & 7) | e / K << 3, kc = e / 8 % (K / 8);
      const uint32_t *s = reinterpret_cast<const uint32_t *>(W + (int64_t)n * K + kc * 8);
      const uint4 v = al ? *reinterpret_cast<const uint4 *>(s) : make_uint4(s[0], s[1], s[2], s[3]);
      *reinterpret_cast<uint4 *>(dst + (n >> 3) * sbo + kc * 128 + (n & 7) * 16) = v;
    }
    return;
  }
  // [k][n]: two k rows of eight columns per thread, paired into words
  const int n8s = N / 8;
#pragma unroll 4
  for (int e = threadIdx.x; e < K / 2 * n8s; e += kMThreads) {
    const int lo = e & 31, hi = e >> 5;
    const int n8 = hi % (n8s / 8) * 8 + (lo >> 2), k = 2 * (hi / (n8s / 8) * 4 + (lo & 3));
    const uint16_t *s0 = W + (int64_t)k * N + n8 * 8, *s1 = s0 + N;
    uint32_t a[4], b[4];
    if (al) {
      const uint4 u = __ldg(reinterpret_cast<const uint4 *>(s0));
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(s1));
      a[0] = u.x, a[1] = u.y, a[2] = u.z, a[3] = u.w;
      b[0] = v.x, b[1] = v.y, b[2] = v.z, b[3] = v.w;
    } else {
      for (int q = 0; q < 4; ++q) {
        a[q] = s0[2 * q] | (uint32_t)s0[2 * q + 1] << 16;
        b[q] = s1[2 * q] | (uint32_t)s1[2 * q + 1] << 16;
      }
    }
    uint8_t *o = dst + n8 * sbo + (k >> 3) * 128 + (k & 7) * 2;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      *reinterpret_cast<uint32_t *>(o + (2 * q) * 16) = __byte_perm(a[q], b[q], 0x5410);
      *reinterpret_cast<uint32_t *>(o + (2 * q + 1) * 16) = __byte_perm(a[q], b[q], 0x7632);
    }
  }
}

// Eight inputs (one core matrix row) of row m as they lie in memory, zero past M.
struct MlpX {
  uint4 u, v;
};
__device__ __forceinline__ MlpX m_load_x(const MlpFwdArgs &A, int64_t m, int kc) {
  MlpX x;
  x.u = x.v = make_uint4(0, 0, 0, 0);
  if (m >= A.M) return x;
  if (A.x32) {
    const uint4 *p = reinterpret_cast<const uint4 *>((const float *)A.X + m * kMIn + kc * 8);
    x.u = p[0], x.v = p[1];
  } else {
    x.u = *reinterpret_cast<const uint4 *>((const uint16_t *)A.X + m * kMIn + kc * 8);
  }
  return x;
}
__device__ __forceinline__ uint4 m_bf16_x(const MlpFwdArgs &A, const MlpX &x) {
  if (!A.x32) return x.u;
  auto two = [](uint32_t lo, uint32_t hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
    return d;
  };
  return make_uint4(two(x.u.x, x.u.y), two(x.u.z, x.u.w), two(x.v.x, x.v.y), two(x.v.z, x.v.w));
}

// A hidden layer's epilogue for this thread's row and 32 columns: the sums at
// `reg` become the next layer's packed A operand in place (KEEP: and, when h is
// given, row-major activations).
template <bool KEEP>
__device__ __forceinline__ void m_epilogue(uint32_t reg, const float *bias, uint16_t *h) {
  uint32_t r[32], p[16];
  m_ld32(r, reg);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float4 bb = *reinterpret_cast<const float4 *>(bias + 4 * q);
    p[2 * q] = m_bias_relu(r[4 * q], r[4 * q + 1], bb.x, bb.y);
    p[2 * q + 1] = m_bias_relu(r[4 * q + 2], r[4 * q + 3], bb.z, bb.w);
  }
  m_st16(reg, p);
#pragma unroll
  for (int q = 0; KEEP && q < 4; ++q)
    m_keep(h ? h + 8 * q : nullptr, p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// The third layer's epilogue and the head of this thread's row: s[l] sums
// columns l, l + 32, l + 64, l + 96, then the butterfly's tree over l.
template <bool KEEP>
__device__ __forceinline__ float m_head(uint32_t reg, const float *b3, const float *w4, uint16_t *h) {
  float s[32];
#pragma unroll
  for (int l = 0; l < 32; ++l) s[l] = 0.f;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    uint32_t r[32];
    m_ld32(r, reg + 32 * c);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 bb = *reinterpret_cast<const float4 *>(b3 + 32 * c + 4 * q);
      const float4 ww = *reinterpret_cast<const float4 *>(w4 + 32 * c + 4 * q);
      r[2 * q] = m_bias_relu(r[4 * q], r[4 * q + 1], bb.x, bb.y);
      r[2 * q + 1] = m_bias_relu(r[4 * q + 2], r[4 * q + 3], bb.z, bb.w);
      s[4 * q] = fmaf(__uint_as_float(r[2 * q] << 16), ww.x, s[4 * q]);
      s[4 * q + 1] = fmaf(__uint_as_float(r[2 * q] & 0xFFFF0000u), ww.y, s[4 * q + 1]);
      s[4 * q + 2] = fmaf(__uint_as_float(r[2 * q + 1] << 16), ww.z, s[4 * q + 2]);
      s[4 * q + 3] = fmaf(__uint_as_float(r[2 * q + 1] & 0xFFFF0000u), ww.w, s[4 * q + 3]);
    }
#pragma unroll
    for (int q = 0; KEEP && q < 4; ++q)
      m_keep(h ? h + 32 * c + 8 * q : nullptr, r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int l = 0; l < o; ++l) s[l] += s[l + o];
  return s[0];
}

// KEEP: the hidden layers' activations are wanted.
template <bool KEEP>
__global__ void __launch_bounds__(kMThreads, 1) k_mlp_forward(const __grid_constant__ MlpFwdArgs A) {
  extern __shared__ unsigned char mlp_raw[];
  uint8_t *sm = mlp_raw + ((128 - ((uint32_t)__cvta_generic_to_shared(mlp_raw) & 127)) & 127);
  const uint32_t sb = (uint32_t)__cvta_generic_to_shared(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int quarter = warp >> 2;                    // columns 32 quarter .. of a half; 4: the head
  const int row = (warp & 3) * 32 + lane;           // this thread's TMEM lane
  float *bias = reinterpret_cast<float *>(sm + kMBias);
  // mbarriers: layers 1, 2, 3 done; the head has read its sums
  const uint32_t bar1 = sb + kMBar, bar2 = bar1 + 8, bar3 = bar1 + 16, bar_head = bar1 + 24;
  uint32_t *slot = reinterpret_cast<uint32_t *>(sm + kMBar + 32);
  volatile int *dead = reinterpret_cast<volatile int *>(sm + kMBar + 40);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(sb + kMBar + 32)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int q = 0; q < 4; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar1 + 8 * q), "r"(q == 3 ? 4 : 1)
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *dead = 0;
  }
  m_stage_w(sm + kMW1, A.W[0], kMIn, kMH1, A.trans);
  m_stage_w(sm + kMW2, A.W[1], kMH1, kMH2, A.trans);
  m_stage_w(sm + kMW3, A.W[2], kMH2, kMH3, A.trans);
  for (int i = tid; i < kMH1 + kMH2 + 2 * kMH3; i += kMThreads)
    bias[i] = i < 256 ? A.b[0][i] : i < 512 ? A.b[1][i - 256] : i < 640 ? A.b[2][i - 512]
              : __uint_as_float((uint32_t)A.w4[i - 640] << 16);
  const int tiles = m_tiles(A.M);
  // a main thread's core matrix row of an input tile
  auto put_x = [&](const MlpX &x) {
    const int r = (tid & 7) | tid >> 5 << 3, kc = tid >> 3 & 3;
    *reinterpret_cast<uint4 *>(sm + kMX + (r >> 3) * m_sbo(kMIn) + kc * 128 + (r & 7) * 16) = m_bf16_x(A, x);
  };
  auto get_x = [&](int t) {
    return m_load_x(A, (int64_t)t * kMRows + ((tid & 7) | tid >> 5 << 3), tid >> 3 & 3);
  };
  if (tid < kMMain && (int)blockIdx.x < tiles) put_x(get_x(blockIdx.x));
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // staged operands
  m_before();
  __syncthreads();
  m_after();
  const uint32_t tm = *slot;
  const uint32_t lane_base = (uint32_t)(warp & 3) << 21;  // TMEM lane 32 (warp % 4) in bits 16-
  auto layer1 = [&](uint32_t d) {
    for (int k = 0; k < kMIn / 16; ++k)
      m_mma_ss(d, m_desc(sb + kMX + 256 * k, m_sbo(kMIn)), m_desc(sb + kMW1 + 256 * k, m_sbo(kMIn)),
               m_idesc(kMH1), k);
    m_commit(bar1);
  };
  // n columns of a layer over half h of its k.  Its packed A: 16 columns of each 32
  // that the sums had
  auto half = [&](uint32_t d, uint32_t a, uint32_t w, int h, int n) {
#pragma unroll
    for (int k = 8 * h; k < 8 * h + 8; ++k)
      m_mma_ts(d, a + 32 * (k >> 1) + 8 * (k & 1), m_desc(sb + w + 256 * k, m_sbo(kMH1)), m_idesc(n), k);
  };
  // A wait that runs out marks the CTA; the main warps leave together after the
  // next barrier, the head's before their next tile.
  auto wait = [&](uint32_t bar, uint32_t parity) {
    if (!m_wait(bar, parity)) *dead = 1;
    m_after();
  };
  uint32_t i = 0;  // tiles done: the barriers' phases, the regions' places
  if (quarter < 4) {
    if (tid == 0 && (int)blockIdx.x < tiles) layer1(tm);
    // the next tile's inputs travel for a whole tile, unconverted
    MlpX x = get_x(blockIdx.x + gridDim.x);
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
      const uint32_t P = tm + 256 * (i & 1), Q = tm + 256 * (~i & 1);
      const uint32_t mine = lane_base + 32 * quarter;
      const float *b1 = bias + 32 * quarter, *b2 = b1 + 256;
      const int tn = t + gridDim.x;
      const int64_t m = (int64_t)t * kMRows + row;
      const bool in = m < A.M;
      uint16_t *h1 = in && A.H[0] ? A.H[0] + m * kMH1 + 32 * quarter : nullptr;
      uint16_t *h2 = in && A.H[1] ? A.H[1] + m * kMH2 + 32 * quarter : nullptr;
      wait(bar1, i & 1);
      put_x(x);
      x = get_x(tn + gridDim.x);
      __syncwarp();
      m_epilogue<KEEP>(P + mine, b1, h1);
      m_before();
      if (m_main_sync(*dead)) break;
      if (tid == 0) {
        if (i) wait(bar_head, ~i & 1);  // the last tile's sums are in Q
        m_after();
        half(Q, P, kMW2, 0, kMH2);
      }
      __syncwarp();
      m_epilogue<KEEP>(P + mine + 128, b1 + 128, h1 ? h1 + 128 : nullptr);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the next inputs
      m_before();
      if (m_main_sync(*dead)) break;
      if (tid == 0) {
        m_after();
        half(Q, P, kMW2, 1, kMH2);
        m_commit(bar2);
      }
      wait(bar2, i & 1);
      __syncwarp();
      m_epilogue<KEEP>(Q + mine, b2, h2);
      m_before();
      if (m_main_sync(*dead)) break;
      if (tid == 0) {
        m_after();
        half(P, Q, kMW3, 0, kMH3);
      }
      __syncwarp();
      m_epilogue<KEEP>(Q + mine + 128, b2 + 128, h2 ? h2 + 128 : nullptr);
      m_before();
      if (m_main_sync(*dead)) break;
      if (tid == 0) {
        m_after();
        half(P, Q, kMW3, 1, kMH3);
        m_commit(bar3);
        wait(bar3, i & 1);
        if (tn < tiles) layer1(Q);
      }
    }
  } else {
    // a warp leaves as one: its lanes may read the mark at different times
    for (int t = blockIdx.x; t < tiles && !__any_sync(0xffffffffu, *dead); t += gridDim.x, ++i) {
      const uint32_t P = tm + 256 * (i & 1);
      const int64_t m = (int64_t)t * kMRows + row;
      const bool in = m < A.M;
      wait(bar3, i & 1);
      __syncwarp();
      const float s = m_head<KEEP>(P + lane_base, bias + 512, bias + 640,
                             in && A.H[2] ? A.H[2] + m * kMH3 : nullptr);
      m_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_head) : "memory");
      if (in) A.y[m] = s + A.b4[0];
    }
  }
  m_before();
  __syncthreads();
  if (*dead)  // a product never completed: no prediction may pass for one
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x)
      if (quarter == 4 && t * kMRows + row < A.M) A.y[t * kMRows + row] = __int_as_float(0x7FFFFFFF);
  if (warp == 0) {
    m_after();
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tm) : "memory");
  }
}

int mlp_forward(const MlpFwdArgs &A, cudaStream_t st) {
  if (A.M < 0) return fail(POYD_EINVAL, "negative size");
  if (A.M == 0) return POYD_OK;
  for (int i = 0; i < 3; ++i)
    if (!A.W[i] || !A.b[i] || ((uintptr_t)A.W[i] & 3) || ((uintptr_t)A.H[i] & 15))
      return fail(POYD_EINVAL, "MLP forward: null or misaligned layer %d", i + 1);
  if (!A.X || !A.w4 || !A.b4 || !A.y) return fail(POYD_EINVAL, "MLP forward: null argument");
  if ((uintptr_t)A.X & 15) return fail(POYD_EINVAL, "MLP forward: X must be 16-byte aligned");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  auto kern = A.H[0] || A.H[1] || A.H[2] ? k_mlp_forward<true> : k_mlp_forward<false>;
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMSmem);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_mlp_forward)");
  const int tiles = m_tiles(A.M);
  {
    ProfScope ps("mlp_forward", st);
    kern<<<tiles < sms ? tiles : sms, kMThreads, kMSmem, st>>>(A);
  }
  const cudaError_t l = cudaGetLastError();
  return l != cudaSuccess ? cuda_fail(l, "k_mlp_forward") : POYD_OK;
}

}  // namespace
}  // namespace poyd

using namespace poyd;

extern "C" int poyd_mlp_forward(const void *X, int32_t M, const void *W1t, const float *b1,
                                const void *W2t, const float *b2, const void *W3t,
                                const float *b3, const void *w4, const float *b4, float *y,
                                void *stream) {
  MlpFwdArgs A = {};
  A.X = X;
  A.trans = 1;
  A.M = M;
  const void *W[3] = {W1t, W2t, W3t};
  const float *b[3] = {b1, b2, b3};
  for (int i = 0; i < 3; ++i) A.W[i] = (const uint16_t *)W[i], A.b[i] = b[i];
  A.w4 = (const uint16_t *)w4;
  A.b4 = b4;
  A.y = y;
  return mlp_forward(A, (cudaStream_t)stream);
}

extern "C" int poyd_mlp_forward_rows(const void *X, int32_t x_fp32, int32_t M, const void *W1,
                                     const float *b1, const void *W2, const float *b2,
                                     const void *W3, const float *b3, const void *w4,
                                     const float *b4, void *H1, void *H2, void *H3, float *y,
                                     void *stream) {
  MlpFwdArgs A = {};
  A.X = X;
  A.x32 = x_fp32;
  A.M = M;
  const void *W[3] = {W1, W2, W3};
  const float *b[3] = {b1, b2, b3};
  void *H[3] = {H1, H2, H3};
  for (int i = 0; i < 3; ++i)
    A.W[i] = (const uint16_t *)W[i], A.b[i] = b[i], A.H[i] = (uint16_t *)H[i];
  A.w4 = (const uint16_t *)w4;
  A.b4 = b4;
  A.y = y;
  return mlp_forward(A, (cudaStream_t)stream);
}
