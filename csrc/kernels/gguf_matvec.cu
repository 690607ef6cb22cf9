// Linear layers and routed experts on RAW GGUF blocks: the quantised weights stay in their
// file layout in HBM and are decoded in registers, eight weights per lane, on their way
// into the FMA. One warp walks one output row (or a gate/up row pair) 256 weights per step.
//
//   pk_gguf_linear   y[m, n] = sum_k x[m, k] W[n, k]        (1..8 rows; bf16 / fp32 / SwiGLU out)
//   pk_gguf_moe_w13  h[route, j] = silu(W1_e x_t) * (W3_e x_t) * route weight
//   pk_gguf_moe_w2   y[t] += W2_e h[route]                   (fp32 atomics, or per-route partials)
//
// Device type ids follow the reference's table (src/loader/gguf/quant_types.py): iq2_xxs 0,
// q2_k 1, iq1_m 2, q4_k 3, q5_k 4, iq2_xs 5, iq3_xxs 6, iq4_xs 7, q6_k 8, plus q8_0 9 and
// bf16 10 here. Replaces its DP4A / float kernels (src/csrc/cuda_kernel_impl.cu:6545-6632,
// 7039-8275: gguf_quant_gemm*, gguf_moe_w13*, gguf_moe_w2*, gguf_moe_single_*).
#include <cooperative_groups.h>
#include <algorithm>
#include <mutex>

#include "../common/pk_common.cuh"

namespace {

using namespace pk;

#include "gguf_codebooks.inc"

enum : int { T_IQ2_XXS = 0, T_Q2_K = 1, T_IQ1_M = 2, T_Q4_K = 3, T_Q5_K = 4, T_IQ2_XS = 5, T_IQ3_XXS = 6,
             T_IQ4_XS = 7, T_Q6_K = 8, T_Q8_0 = 9, T_BF16 = 10, T_MXFP4 = 11 };
constexpr int T_LAST = T_MXFP4;

__host__ __device__ constexpr int block_bytes(int t) {
  return t == T_IQ2_XXS ? 66 : t == T_Q2_K ? 84 : t == T_IQ1_M ? 56 : t == T_Q4_K ? 144 : t == T_Q5_K ? 176
       : t == T_IQ2_XS ? 74 : t == T_IQ3_XXS ? 98 : t == T_IQ4_XS ? 136 : t == T_Q6_K ? 210 : t == T_Q8_0 ? 272 : t == T_MXFP4 ? 136 : 512;
}

__device__ __forceinline__ float ld_f16(const uint8_t* p) {
  const uint16_t v = (uint16_t)p[0] | ((uint16_t)p[1] << 8);
  return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ uint32_t ld_u32(const uint8_t* p) {
  return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
}
__device__ __forceinline__ uint32_t ld_u16(const uint8_t* p) { return (uint32_t)p[0] | ((uint32_t)p[1] << 8); }

__device__ __forceinline__ void k4_scale_min(const uint8_t* s, int j, float& sc, float& mn) {
  if (j < 4) {
    sc = (float)(s[j] & 63);
    mn = (float)(s[j + 4] & 63);
  } else {
    sc = (float)((s[j + 4] & 15) | ((s[j - 4] >> 6) << 4));
    mn = (float)((s[j + 4] >> 4) | ((s[j] >> 6) << 4));
  }
}

__device__ const float kIq4nl[16] = {-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113};

// Weights [8p, 8p + 8) of one 256-weight super block (for q8_0: eight 34-byte blocks).
template <int TYPE>
__device__ __forceinline__ void decode8(const uint8_t* b, int p, float (&w)[8]) {
  if constexpr (TYPE == T_Q8_0) {
    const uint8_t* blk = b + (p >> 2) * 34;
    const float d = ld_f16(blk);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = d * (float)(int8_t)blk[2 + (p & 3) * 8 + i];
  } else if constexpr (TYPE == T_BF16) {
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = __uint_as_float(ld_u16(b + (p * 8 + i) * 2) << 16);
  } else if constexpr (TYPE == T_MXFP4) {
    // eight 17-byte groups: one E8M0 scale, then 32 E2M1 nibbles (element 2j low, 2j+1 high)
    const uint8_t* blk = b + (p >> 2) * 17;
    const float d = e8m0_to_float(blk[0]);
    const uint8_t* q = blk + 1 + (p & 3) * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[2 * i] = d * e2m1_to_float(q[i] & 15);
      w[2 * i + 1] = d * e2m1_to_float(q[i] >> 4);
    }
  } else if constexpr (TYPE == T_Q2_K) {
    const int g = p >> 1, half = g >> 3, gi = g & 7, shift = (gi >> 1) * 2;
    const uint8_t* q = b + 16 + half * 32 + (gi & 1) * 16 + (p & 1) * 8;
    const uint8_t s = b[g];
    const float d = ld_f16(b + 80) * (float)(s & 15), m = ld_f16(b + 82) * (float)(s >> 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = d * (float)((q[i] >> shift) & 3) - m;
  } else if constexpr (TYPE == T_Q4_K || TYPE == T_Q5_K) {
    const int pr = p >> 3, h = (p >> 2) & 1, l0 = (p & 3) * 8, j = 2 * pr + h;
    float sc, mn;
    k4_scale_min(b + 4, j, sc, mn);
    const float d = ld_f16(b) * sc, m = ld_f16(b + 2) * mn;
    const uint8_t* q = b + (TYPE == T_Q4_K ? 16 : 48) + pr * 32 + l0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int v = h ? (q[i] >> 4) : (q[i] & 15);
      if constexpr (TYPE == T_Q5_K) v += ((b[16 + l0 + i] >> j) & 1) << 4;
      w[i] = d * (float)v - m;
    }
  } else if constexpr (TYPE == T_Q6_K) {
    const int n = p >> 4, idx = (p & 15) * 8, k = idx >> 5, l0 = idx & 31;
    const uint8_t* ql = b + 64 * n + (k & 1) * 32 + l0;
    const uint8_t* qh = b + 128 + 32 * n + l0;
    const float d = ld_f16(b + 208) * (float)(int8_t)b[192 + 8 * n + 2 * k + (l0 >> 4)];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int lo = k < 2 ? (ql[i] & 15) : (ql[i] >> 4);
      w[i] = d * (float)((lo | (((qh[i] >> (2 * k)) & 3) << 4)) - 32);
    }
  } else if constexpr (TYPE == T_IQ2_XXS) {
    const int sub = p >> 2, part = p & 3;
    const uint8_t* q = b + 2 + sub * 8;
    const uint32_t aux = ld_u32(q + 4);
    const float d = ld_f16(b) * 0.125f * (float)(2 * (aux >> 28) + 1);
    const uint64_t g = kIq2xxsGrid[q[part]];
    const uint8_t sg = kKsigns[(aux >> (7 * part)) & 127];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float v = d * (float)((g >> (8 * i)) & 0xff);
      w[i] = (sg >> i) & 1 ? -v : v;
    }
  } else if constexpr (TYPE == T_IQ2_XS) {
    const int sub = p >> 2, part = p & 3;
    const uint32_t q = ld_u16(b + 2 + (sub * 4 + part) * 2);
    const uint32_t nib = (b[66 + sub] >> (4 * (part >> 1))) & 15;
    const float d = ld_f16(b) * 0.25f * ((float)nib + 0.5f);
    const uint64_t g = kIq2xsGrid[q & 511];
    const uint8_t sg = kKsigns[q >> 9];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float v = d * (float)((g >> (8 * i)) & 0xff);
      w[i] = (sg >> i) & 1 ? -v : v;
    }
  } else if constexpr (TYPE == T_IQ3_XXS) {
    const int sub = p >> 2, pr = p & 3;
    const uint32_t aux = ld_u32(b + 66 + sub * 4);
    const float d = ld_f16(b) * 0.5f * ((float)(aux >> 28) + 0.5f);
    const uint32_t g0 = kIq3xxsGrid[b[2 + sub * 8 + pr * 2]], g1 = kIq3xxsGrid[b[2 + sub * 8 + pr * 2 + 1]];
    const uint8_t sg = kKsigns[(aux >> (7 * pr)) & 127];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float v0 = d * (float)((g0 >> (8 * i)) & 0xff), v1 = d * (float)((g1 >> (8 * i)) & 0xff);
      w[i] = (sg >> i) & 1 ? -v0 : v0;
      w[4 + i] = (sg >> (4 + i)) & 1 ? -v1 : v1;
    }
  } else if constexpr (TYPE == T_IQ4_XS) {
    const int ib = p >> 2, q = p & 3;
    const uint32_t sh = ld_u16(b + 2);
    const int ls = ((b[4 + (ib >> 1)] >> (4 * (ib & 1))) & 15) | (((sh >> (2 * ib)) & 3) << 4);
    const float d = ld_f16(b) * (float)(ls - 32);
    const uint8_t* qs = b + 8 + 16 * ib + 8 * (q & 1);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = d * kIq4nl[q < 2 ? (qs[i] & 15) : (qs[i] >> 4)];
  } else if constexpr (TYPE == T_IQ1_M) {
    const int ib = p >> 2, g = p & 3;
    const uint32_t s0 = ld_u16(b + 48), s1 = ld_u16(b + 50), s2 = ld_u16(b + 52), s3 = ld_u16(b + 54);
    const uint16_t dbits = (uint16_t)((s0 >> 12) | ((s1 >> 8) & 0xf0) | ((s2 >> 4) & 0xf00) | (s3 & 0xf000));
    const uint32_t sw = ld_u16(b + 48 + (ib >> 1) * 2) >> (6 * (ib & 1));
    const float dl = __half2float(__ushort_as_half(dbits)) * (float)(2 * ((sw >> (3 * (g >> 1))) & 7) + 1);
    const uint32_t h = b[32 + 2 * ib + (g >> 1)];
    const uint32_t idx = b[4 * ib + g] | (((g & 1) ? (h << 4) : (h << 8)) & 0x700);
    const float delta = (h & ((g & 1) ? 0x80 : 0x08)) ? -0.125f : 0.125f;
    const uint64_t gr = kIq1Grid[idx];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = dl * ((float)(int8_t)((gr >> (8 * i)) & 0xff) + delta);
  }
}

constexpr int kThreads = 256;
constexpr int kWarps = 8;

// The decoders read single bytes; from global memory that is one load instruction per byte, each a round trip to L2.
// A warp therefore first brings a stretch of its row into shared memory with 16-byte loads and decodes from there.
constexpr int kStageBlocks = 8;                                  // 2048 weights per stretch
// Bytes of one warp's stage buffer for rows of `type` with K weights: a stretch of up to kStageBlocks blocks plus the
// misalignment of its start, rounded to 16. Sized per launch so that small block types leave room for more resident blocks.
__host__ __device__ inline int stage_bytes_per_warp(int type, int K) {
  const int nb = (K >> 8) < kStageBlocks ? (K >> 8) : kStageBlocks;
  return ((nb * block_bytes(type) + 15) & ~15) + 16;
}

// One warp: dot products of one raw row with M staged activation rows (fp32, [M][K]). `stage` is this warp's
// stage_bytes_per_warp(TYPE, K) bytes of shared memory.
template <int TYPE, int M>
__device__ __forceinline__ void row_dot(const uint8_t* wrow, const float* xs, int K, int lane, float (&acc)[M], uint8_t* stage) {
  constexpr int BB = block_bytes(TYPE);
  const int nblk = K >> 8;
  if (stage == nullptr) {
    // Several activation rows share every decoded weight, which hides the byte loads: decode straight from global memory
    // (and keep the shared memory for a second resident block).
    for (int blk = 0; blk < nblk; ++blk) {
      float w[8];
      decode8<TYPE>(wrow + (size_t)blk * BB, lane, w);
      const int k = (blk << 8) + (lane << 3);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(xs + m * K + k);
        const float4 c = *reinterpret_cast<const float4*>(xs + m * K + k + 4);
        acc[m] += w[0] * a.x + w[1] * a.y + w[2] * a.z + w[3] * a.w + w[4] * c.x + w[5] * c.y + w[6] * c.z + w[7] * c.w;
      }
    }
    return;
  }
  for (int blk0 = 0; blk0 < nblk; blk0 += kStageBlocks) {
    const int nb = min(kStageBlocks, nblk - blk0);
    const uint8_t* src = wrow + (size_t)blk0 * BB;
    const int mis = (int)((uintptr_t)src & 15);
    const uint8_t* src_al = src - mis;           // the bytes before `src` belong to the previous row or block of the same tensor
    const int total = mis + nb * BB;
    __syncwarp();                                // the previous stretch has been decoded by every lane
    for (int off = lane << 4; off < total; off += 512) {
      if (off + 16 <= total) {
        *reinterpret_cast<uint4*>(stage + off) = __ldg(reinterpret_cast<const uint4*>(src_al + off));
      } else {
        for (int i = off < mis ? mis - off : 0; off + i < total; ++i) stage[off + i] = src_al[off + i];   // never past the row's end
      }
    }
    __syncwarp();
    for (int b = 0; b < nb; ++b) {
      float w[8];
      decode8<TYPE>(stage + mis + b * BB, lane, w);
      const int k = ((blk0 + b) << 8) + (lane << 3);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(xs + m * K + k);
        const float4 c = *reinterpret_cast<const float4*>(xs + m * K + k + 4);
        acc[m] += w[0] * a.x + w[1] * a.y + w[2] * a.z + w[3] * a.w + w[4] * c.x + w[5] * c.y + w[6] * c.z + w[7] * c.w;
      }
    }
  }
}

struct LinearParams {
  const uint8_t* W;   // [N, K/256 blocks]
  int type, N, K, M;
  const bf16* x;      // [M, K]
  const float* gamma; // optional fused RMSNorm (plain gamma)
  float eps;
  int epi;            // 0 bf16, 1 swiglu (rows j and j + N/2), 2 fp32
  void* y;
  int ldy;
  int stage_bytes;    // per warp, behind the staged activations in dynamic shared memory (one- and two-row launches)
};

template <int M>
__device__ __forceinline__ void dispatch_row(int type, const uint8_t* wrow, const float* xs, int K, int lane, float (&acc)[M], uint8_t* stage) {
  switch (type) {
    case T_IQ2_XXS: row_dot<T_IQ2_XXS, M>(wrow, xs, K, lane, acc, stage); break;
    case T_Q2_K: row_dot<T_Q2_K, M>(wrow, xs, K, lane, acc, stage); break;
    case T_IQ1_M: row_dot<T_IQ1_M, M>(wrow, xs, K, lane, acc, stage); break;
    case T_Q4_K: row_dot<T_Q4_K, M>(wrow, xs, K, lane, acc, stage); break;
    case T_Q5_K: row_dot<T_Q5_K, M>(wrow, xs, K, lane, acc, stage); break;
    case T_IQ2_XS: row_dot<T_IQ2_XS, M>(wrow, xs, K, lane, acc, stage); break;
    case T_IQ3_XXS: row_dot<T_IQ3_XXS, M>(wrow, xs, K, lane, acc, stage); break;
    case T_IQ4_XS: row_dot<T_IQ4_XS, M>(wrow, xs, K, lane, acc, stage); break;
    case T_Q6_K: row_dot<T_Q6_K, M>(wrow, xs, K, lane, acc, stage); break;
    case T_Q8_0: row_dot<T_Q8_0, M>(wrow, xs, K, lane, acc, stage); break;
    case T_MXFP4: row_dot<T_MXFP4, M>(wrow, xs, K, lane, acc, stage); break;
    default: row_dot<T_BF16, M>(wrow, xs, K, lane, acc, stage); break;
  }
}

__host__ __device__ inline size_t row_bytes(int type, int K) { return (size_t)(K >> 8) * block_bytes(type); }

template <int M>
__global__ void __launch_bounds__(kThreads) gguf_linear_kernel(const LinearParams p) {
  extern __shared__ __align__(16) float xs[];  // [M][K]
  __shared__ float red[40];
  constexpr bool kStaged = M <= 2;     // one or two rows: the byte loads of the decoders dominate, stage the weights
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint8_t* stage = kStaged ? reinterpret_cast<uint8_t*>(xs + (size_t)M * p.K) + (size_t)warp * p.stage_bytes : nullptr;
  for (int m = 0; m < M; ++m) {
    float ss = 0.f;
    for (int k = tid; k < p.K; k += kThreads) {
      // the template may be wider than the number of rows given: pad with zeros
      const float v = m < p.M ? __bfloat162float(p.x[(size_t)m * p.K + k]) : 0.f;
      xs[m * p.K + k] = v;
      ss += v * v;
    }
    if (p.gamma != nullptr) {
      ss = block_sum(ss, red);
      const float rs = rsqrtf(ss / (float)p.K + p.eps);
      for (int k = tid; k < p.K; k += kThreads)
        xs[m * p.K + k] = __bfloat162float(__float2bfloat16(xs[m * p.K + k] * rs * p.gamma[k]));
    }
  }
  __syncthreads();
  const size_t rb = row_bytes(p.type, p.K);
  const int half_n = p.N >> 1;
  const int groups = p.epi == 1 ? half_n : p.N;
  for (int g = blockIdx.x * kWarps + warp; g < groups; g += gridDim.x * kWarps) {
    float a0[M], a1[M];
#pragma unroll
    for (int m = 0; m < M; ++m) { a0[m] = 0.f; a1[m] = 0.f; }
    dispatch_row<M>(p.type, p.W + (size_t)g * rb, xs, p.K, lane, a0, stage);
    if (p.epi == 1) dispatch_row<M>(p.type, p.W + (size_t)(g + half_n) * rb, xs, p.K, lane, a1, stage);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      a0[m] = warp_sum(a0[m]);
      if (p.epi == 1) a1[m] = warp_sum(a1[m]);
    }
    if (lane == 0) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        if (m >= p.M) break;
        if (p.epi == 1) ((bf16*)p.y)[(size_t)m * p.ldy + g] = __float2bfloat16(silu(a0[m]) * a1[m]);
        else if (p.epi == 0) ((bf16*)p.y)[(size_t)m * p.ldy + g] = __float2bfloat16(a0[m]);
        else ((float*)p.y)[(size_t)m * p.ldy + g] = a0[m];
      }
    }
  }
}

// ---- routed experts ----
// Routes are sorted by expert: seg_start[e] .. seg_start[e+1] index into route_token / route_weight.
constexpr int kRouteParallelMax = 64;   // up to this many routes in a step, every route gets its own blocks

struct MoeParams {
  const uint8_t* W13;  // [E, 2I, H] raw rows (gate rows then up rows per expert)
  const uint8_t* W2;   // [E, H, I]
  int type13, type2;
  int E, H, I;
  const bf16* x;        // [T, H]
  const int* seg_start; // [E + 1]
  const int* route_token;   // [R]
  const float* route_weight; // [R]
  float* hbuf;          // [R, I] fp32 hidden of every route (already times the route weight)
  float* y;             // [T, H] fp32, accumulated with atomics
  float limit;          // SwiGLU clamp, 0 = off
  int expert_offset;    // first expert id stored in W13 / W2 (expert parallel shard)
  int local_experts;
  float* ybuf;          // [R, H] per-route outputs for the fixed-order reduce; null = atomics into y
};

// Gate/up rows of one expert against MB staged tokens (MB = 1, 2, 4 or 8: a decode step has one token per expert, and
// decoding a weight once per token slot that is not there would be wasted arithmetic).
template <int MB>
__device__ __forceinline__ void moe_w13_rows(const MoeParams& p, const uint8_t* base, size_t rb, const float* xs, int rs, int cnt, int lane,
                                             int warp, uint8_t* stage) {
  for (int j = blockIdx.x * kWarps + warp; j < p.I; j += gridDim.x * kWarps) {
    float g[MB], u[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) { g[m] = 0.f; u[m] = 0.f; }
    dispatch_row<MB>(p.type13, base + (size_t)j * rb, xs, p.H, lane, g, stage);
    dispatch_row<MB>(p.type13, base + (size_t)(p.I + j) * rb, xs, p.H, lane, u, stage);
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      float gv = warp_sum(g[m]), uv = warp_sum(u[m]);
      if (p.limit > 0.f) {
        gv = fminf(gv, p.limit);
        uv = fminf(fmaxf(uv, -p.limit), p.limit);
      }
      if (lane == 0 && m < cnt) p.hbuf[(size_t)(rs + m) * p.I + j] = silu(gv) * uv * p.route_weight[rs + m];
    }
  }
}

template <int MB>
__device__ __forceinline__ void moe_w2_rows(const MoeParams& p, const uint8_t* base, size_t rb, const float* hs, int rs, int cnt, int lane,
                                            int warp, uint8_t* stage) {
  for (int n = blockIdx.x * kWarps + warp; n < p.H; n += gridDim.x * kWarps) {
    float a[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) a[m] = 0.f;
    dispatch_row<MB>(p.type2, base + (size_t)n * rb, hs, p.I, lane, a, stage);
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const float v = warp_sum(a[m]);
      if (lane == 0 && m < cnt) {
        if (p.ybuf != nullptr) p.ybuf[(size_t)(rs + m) * p.H + n] = v;
        else atomicAdd(p.y + (size_t)p.route_token[rs + m] * p.H + n, v);
      }
    }
  }
}

// grid: (row tiles, local experts). Each block stages up to 8 routed tokens of its expert at a
// time and lets its warps walk gate/up row pairs.
__global__ void __launch_bounds__(kThreads) gguf_moe_w13_kernel(const MoeParams p) {
  extern __shared__ __align__(16) float xs[];  // [8][H]
  const int le = blockIdx.y, e = le + p.expert_offset;
  const int r0 = p.seg_start[e], r1 = p.seg_start[e + 1];
  if (r0 >= r1) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t rb = row_bytes(p.type13, p.H);
  const uint8_t* base = p.W13 + (size_t)le * 2 * p.I * rb;
  for (int rs = r0; rs < r1; rs += 8) {
    const int cnt = min(8, r1 - rs);
    __syncthreads();
    const int mb = cnt <= 1 ? 1 : cnt <= 2 ? 2 : cnt <= 4 ? 4 : 8;
    for (int m = 0; m < mb; ++m)
      for (int k = tid; k < p.H; k += kThreads)
        xs[m * p.H + k] = m < cnt ? __bfloat162float(p.x[(size_t)p.route_token[rs + m] * p.H + k]) : 0.f;
    __syncthreads();
    if (mb == 1) moe_w13_rows<1>(p, base, rb, xs, rs, cnt, lane, warp, nullptr);
    else if (mb == 2) moe_w13_rows<2>(p, base, rb, xs, rs, cnt, lane, warp, nullptr);
    else if (mb == 4) moe_w13_rows<4>(p, base, rb, xs, rs, cnt, lane, warp, nullptr);
    else moe_w13_rows<8>(p, base, rb, xs, rs, cnt, lane, warp, nullptr);
  }
}

__global__ void __launch_bounds__(kThreads) gguf_moe_w2_kernel(const MoeParams p) {
  extern __shared__ __align__(16) float hs[];  // [8][I]
  const int le = blockIdx.y, e = le + p.expert_offset;
  const int r0 = p.seg_start[e], r1 = p.seg_start[e + 1];
  if (r0 >= r1) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t rb = row_bytes(p.type2, p.I);
  const uint8_t* base = p.W2 + (size_t)le * p.H * rb;
  for (int rs = r0; rs < r1; rs += 8) {
    const int cnt = min(8, r1 - rs);
    __syncthreads();
    const int mb = cnt <= 1 ? 1 : cnt <= 2 ? 2 : cnt <= 4 ? 4 : 8;
    for (int m = 0; m < mb; ++m)
      for (int k = tid; k < p.I; k += kThreads) hs[m * p.I + k] = m < cnt ? p.hbuf[(size_t)(rs + m) * p.I + k] : 0.f;
    __syncthreads();
    if (mb == 1) moe_w2_rows<1>(p, base, rb, hs, rs, cnt, lane, warp, nullptr);
    else if (mb == 2) moe_w2_rows<2>(p, base, rb, hs, rs, cnt, lane, warp, nullptr);
    else if (mb == 4) moe_w2_rows<4>(p, base, rb, hs, rs, cnt, lane, warp, nullptr);
    else moe_w2_rows<8>(p, base, rb, hs, rs, cnt, lane, warp, nullptr);
  }
}

// Few routes (decode, speculative verify): grid (row tiles, routes of this rank). Every block serves ONE route, so all
// blocks have work and an expert's rows spread over as many blocks as there are tiles; the expert of a route comes
// from a binary search in seg_start.
__device__ __forceinline__ int expert_of_route(const int* seg_start, int lo_e, int hi_e, int r) {
  while (hi_e - lo_e > 1) {   // invariant: seg_start[lo_e] <= r < seg_start[hi_e]
    const int mid = (lo_e + hi_e) >> 1;
    if (seg_start[mid] <= r) lo_e = mid;
    else hi_e = mid;
  }
  return lo_e;
}

__global__ void __launch_bounds__(kThreads) gguf_moe_w13_route_kernel(const MoeParams p) {
  extern __shared__ __align__(16) float xs[];  // [H], then the warps' stage buffers
  const int lo = p.seg_start[p.expert_offset], hi = p.seg_start[p.expert_offset + p.local_experts];
  const int r = lo + blockIdx.y;
  if (r >= hi) return;
  const int e = expert_of_route(p.seg_start, p.expert_offset, p.expert_offset + p.local_experts, r);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t rb = row_bytes(p.type13, p.H);
  const uint8_t* base = p.W13 + (size_t)(e - p.expert_offset) * 2 * p.I * rb;
  for (int k = tid; k < p.H; k += kThreads) xs[k] = __bfloat162float(p.x[(size_t)p.route_token[r] * p.H + k]);
  __syncthreads();
  moe_w13_rows<1>(p, base, rb, xs, r, 1, lane, warp,
                  reinterpret_cast<uint8_t*>(xs + p.H) + (size_t)warp * stage_bytes_per_warp(p.type13, p.H));
}

__global__ void __launch_bounds__(kThreads) gguf_moe_w2_route_kernel(const MoeParams p) {
  extern __shared__ __align__(16) float hs[];  // [I], then the warps' stage buffers
  const int lo = p.seg_start[p.expert_offset], hi = p.seg_start[p.expert_offset + p.local_experts];
  const int r = lo + blockIdx.y;
  if (r >= hi) return;
  const int e = expert_of_route(p.seg_start, p.expert_offset, p.expert_offset + p.local_experts, r);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t rb = row_bytes(p.type2, p.I);
  const uint8_t* base = p.W2 + (size_t)(e - p.expert_offset) * p.H * rb;
  for (int k = tid; k < p.I; k += kThreads) hs[k] = p.hbuf[(size_t)r * p.I + k];
  __syncthreads();
  moe_w2_rows<1>(p, base, rb, hs, r, 1, lane, warp,
                 reinterpret_cast<uint8_t*>(hs + p.I) + (size_t)warp * stage_bytes_per_warp(p.type2, p.I));
}

// Fixed-order reduce: y[t] += sum over k = 0..topk-1 of the output of route (t, k), skipping routes whose
// expert lives on another rank. route_pos[t * topk + k] is the route's position in the expert-sorted order.
__global__ void moe_reduce_routes_kernel(const float* __restrict__ ybuf, const int* __restrict__ route_pos, const int* __restrict__ seg_start,
                                         int topk, int H, int expert_offset, int local_experts, float* y) {
  const int t = blockIdx.y, n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= H) return;
  const int lo = seg_start[expert_offset], hi = seg_start[expert_offset + local_experts];
  float acc = y[(size_t)t * H + n];
  for (int k = 0; k < topk; ++k) {
    const int pos = route_pos[t * topk + k];
    if (pos >= lo && pos < hi) acc += ybuf[(size_t)pos * H + n];
  }
  y[(size_t)t * H + n] = acc;
}

// The same reduce with the route weight applied here (ybuf holds unweighted expert outputs, e.g. from the grouped GEMM).
__global__ void moe_reduce_routes_weighted_kernel(const float* __restrict__ ybuf, const float* __restrict__ route_weight,
                                                  const int* __restrict__ route_pos, const int* __restrict__ seg_start, int topk, int H,
                                                  int expert_offset, int local_experts, float* y) {
  pk::pdl_wait_for(ybuf, route_weight, route_pos, seg_start);
  pk::pdl_trigger();
  const int t = blockIdx.y, n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= H) return;
  const int lo = seg_start[expert_offset], hi = seg_start[expert_offset + local_experts];
  float acc = y[(size_t)t * H + n];
  for (int k = 0; k < topk; ++k) {
    const int pos = route_pos[t * topk + k];
    if (pos >= lo && pos < hi) acc = fmaf(route_weight[pos], ybuf[(size_t)pos * H + n], acc);
  }
  y[(size_t)t * H + n] = acc;
}

__global__ void invert_routes_kernel(const int* __restrict__ route_src, int R, int* route_pos) {
  pk::pdl_wait_for(route_src);
  pk::pdl_trigger();
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos < R) route_pos[route_src[pos]] = pos;
}

// ---- routing ----
// Router logits: grid (expert groups of 8, token tiles of up to 8); one warp per expert, which reads its weight row
// once for the tile's tokens. A single token spreads over E / 8 blocks instead of streaming the whole router matrix
// through one block.
__global__ void __launch_bounds__(256) router_logits_kernel(const bf16* x, const float* rw, int H, int E, int T, float* logits) {
  pk::pdl_wait();
  pk::pdl_trigger();
  extern __shared__ __align__(16) float xs[];  // [tokens of the tile][H]
  const int t0 = blockIdx.y * 8, nt = min(8, T - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int m = 0; m < nt; ++m)
    for (int k = tid; k < H; k += 256) xs[m * H + k] = __bfloat162float(x[(size_t)(t0 + m) * H + k]);
  __syncthreads();
  const int e = blockIdx.x * 8 + warp;
  if (e >= E) return;
  float a[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) a[m] = 0.f;
  const float* w = rw + (size_t)e * H;
  const bool vec = (H & 3) == 0 && ((uintptr_t)rw & 15) == 0;
  // one token without the loop over eight: the same sums in the same order
  if (nt == 1 && vec) {
#pragma unroll 8
    for (int k = lane * 4; k < H; k += 128) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(w + k));
      const float4 b = *reinterpret_cast<const float4*>(xs + k);
      a[0] = fmaf(v.w, b.w, fmaf(v.z, b.z, fmaf(v.y, b.y, fmaf(v.x, b.x, a[0]))));
    }
  } else if (nt == 1) {
    for (int k = lane; k < H; k += 32) a[0] = fmaf(w[k], xs[k], a[0]);
  } else if (vec) {
    // by 16 bytes instead of four, 256 experts of 3072: 23 tokens 26.8 -> 18.9 us
#pragma unroll 4
    for (int k = lane * 4; k < H; k += 128) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(w + k));
#pragma unroll
      for (int m = 0; m < 8; ++m)
        if (m < nt) {
          const float4 b = *reinterpret_cast<const float4*>(xs + m * H + k);
          a[m] = fmaf(v.w, b.w, fmaf(v.z, b.z, fmaf(v.y, b.y, fmaf(v.x, b.x, a[m]))));
        }
    }
  } else {
    for (int k = lane; k < H; k += 32) {
      const float wv = w[k];
#pragma unroll
      for (int m = 0; m < 8; ++m)
        if (m < nt) a[m] = fmaf(wv, xs[m * H + k], a[m]);
    }
  }
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    if (m >= nt) break;
    const float v = warp_sum(a[m]);
    if (lane == 0) logits[(size_t)(t0 + m) * E + e] = v;
  }
}

// The same for many tokens: a block has 64 tokens x 64 experts, a thread 8 x 8 sums: 16 reads of shared memory then feed 128
// multiply-adds, which bound it. Four groups of 64 threads take a quarter of every 64 values of K each; where the tiles leave SMs idle the
// blocks of a cluster take a part of K each. All add up in their order (another one than above). Rows come by 16-byte copies where
// they are aligned to that (V = 8), by 4-byte copies where the rows of x are aligned to them (V = 2), and with rows of x at odd addresses those wait in
// registers while a step is multiplied (V = 1). 256 experts, 512 tokens, us: H = 3072 33, 3070 44, 3071 54 (2 x 4 sums a thread 63 each).
// 1500 tokens of 3072 by 256 experts: 73 us (2 x 4 sums a thread, 16 tokens a block: 174; the form above, which reads
// the router's rows once per 8 tokens, 279). 56 % of the rate of fp32 multiply-adds, with one or two blocks on an SM alike.
constexpr int kRt = 64, kRe = 64, kRk = 64, kRs = 3;      // tile, values of K per step, steps in shared memory
constexpr int kRw = kRk + 4, kRx = kRk + 8, kRo = kRe + 8;      // pitches: rows of eight consecutive threads start in different banks
constexpr int kRouterSmem = kRs * (kRe * kRw * 4 + kRt * kRx * 2);
static_assert(4 * kRt * kRo * 4 <= kRouterSmem, "the groups' sums take the place of the tiles");
template <int B>
__device__ __forceinline__ void router_copy(void* dst, const void* src, bool in) {      // B bytes, zeros unless `in`
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst), n = in ? B : 0;
  if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
template <int V>
__global__ void __launch_bounds__(256, 2) router_logits_tile_kernel(const bf16* x, const float* rw, int H, int E, int T, float* logits) {
  extern __shared__ __align__(16) uint8_t router_smem[];
  float* ws = reinterpret_cast<float*>(router_smem);                            // [kRs][kRe][kRw]
  bf16* xs = reinterpret_cast<bf16*>(router_smem + kRs * kRe * kRw * 4);        // [kRs][kRt][kRx]
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int parts = gridDim.x, part = blockIdx.x;      // a cluster is one tile
  const int tid = threadIdx.x, lane = tid & 31, grp = tid >> 6, tx = lane & 7, ty = (lane >> 3) + 4 * ((tid >> 5) & 1);
  const int e0 = blockIdx.y * kRe, t0 = blockIdx.z * kRt;
  const int steps = (H + kRk - 1) / kRk, per = (steps + parts - 1) / parts;
  const int first = min(part * per, steps), n = min(per, steps - first);
  constexpr int WV = V == 8 ? 4 : 1;      // floats of a copy
  auto fetch_w = [&](int i) {
    float* dst = ws + (i % kRs) * kRe * kRw;
    const int k0 = (first + i) * kRk;
#pragma unroll 1
    for (int c = tid; c < kRe * (kRk / WV); c += 256) {
      const int r = c / (kRk / WV), k = (c & (kRk / WV - 1)) * WV;
      const bool in = e0 + r < E && k0 + k < H;
      router_copy<4 * WV>(dst + r * kRw + k, in ? rw + (size_t)(e0 + r) * H + k0 + k : rw, in);
    }
  };
  auto fetch_x = [&](int i) {
    if constexpr (V > 1) {
      bf16* dst = xs + (i % kRs) * kRt * kRx;
      const int k0 = (first + i) * kRk;
#pragma unroll 1
      for (int c = tid; c < kRt * (kRk / V); c += 256) {
        const int r = c / (kRk / V), k = (c & (kRk / V - 1)) * V;
        const bool in = t0 + r < T && k0 + k < H;
        router_copy<2 * V>(dst + r * kRx + k, in ? x + (size_t)(t0 + r) * H + k0 + k : x, in);
      }
    }
  };
  // V = 1: element tid & 63 of every fourth row, two rows in a register
  uint32_t held[V == 1 ? 8 : 1];
  auto load_x = [&](int i) {
    if constexpr (V == 1) {
      const int k = (first + i) * kRk + (tid & 63);
      auto at = [&](int r) -> uint32_t { return t0 + r < T && k < H ? reinterpret_cast<const uint16_t*>(x)[(size_t)(t0 + r) * H + k] : 0; };
#pragma unroll
      for (int j = 0; j < 8; ++j) held[j] = at(grp + 8 * j) | at(grp + 8 * j + 4) << 16;
    }
  };
  auto store_x = [&](int i) {
    if constexpr (V == 1) {
      uint16_t* dst = reinterpret_cast<uint16_t*>(xs) + (i % kRs) * kRt * kRx + (tid & 63);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        dst[(grp + 8 * j) * kRx] = (uint16_t)held[j];
        dst[(grp + 8 * j + 4) * kRx] = (uint16_t)(held[j] >> 16);
      }
    }
  };
  pk::pdl_wait_for(x, rw);      // the router's rows can be the result of the launch before, too
  pk::pdl_trigger();
  for (int i = 0; i < kRs - 1; ++i) {
    if (i < n) {
      fetch_w(i);
      fetch_x(i);
      load_x(i);
      store_x(i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float2 acc[4][8] = {};      // tokens ty + 16 m and ty + 16 m + 8
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kRs - 2) : "memory");
    __syncthreads();
    if (i + kRs - 1 < n) {      // into the buffer that all have read before this barrier
      fetch_w(i + kRs - 1);
      fetch_x(i + kRs - 1);
      load_x(i + kRs - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* w = ws + (i % kRs) * kRe * kRw + tx * kRw + grp * 16;
    const bf16* a = xs + (i % kRs) * kRt * kRx + ty * kRx + grp * 16;
#pragma unroll 2
    for (int k = 0; k < 16; k += 2) {      // two values at a time and no more unrolled: the sums would spill
      float2 v[4][2];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t u = *reinterpret_cast<const uint32_t*>(a + m * 16 * kRx + k), l = *reinterpret_cast<const uint32_t*>(a + (m * 16 + 8) * kRx + k);
        v[m][0] = make_float2(__uint_as_float(u << 16), __uint_as_float(l << 16));
        v[m][1] = make_float2(__uint_as_float(u & 0xffff0000u), __uint_as_float(l & 0xffff0000u));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 b = *reinterpret_cast<const float2*>(w + j * 8 * kRw + k);
#pragma unroll
        for (int m = 0; m < 4; ++m) acc[m][j] = __ffma2_rn(make_float2(b.y, b.y), v[m][1], __ffma2_rn(make_float2(b.x, b.x), v[m][0], acc[m][j]));
      }
    }
    if (i + kRs - 1 < n) store_x(i + kRs - 1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* sums = ws;      // [4][kRt][kRo]
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      sums[(grp * kRt + ty + 16 * m) * kRo + tx + 8 * j] = acc[m][j].x;
      sums[(grp * kRt + ty + 16 * m + 8) * kRo + tx + 8 * j] = acc[m][j].y;
    }
  __syncthreads();
  for (int o = tid; o < kRt * kRe; o += 256) {
    const int r = o / kRe, e = o - r * kRe, at = r * kRo + e;
    const float v = (sums[at] + sums[kRt * kRo + at]) + (sums[2 * kRt * kRo + at] + sums[3 * kRt * kRo + at]);
    if (parts > 1)
      sums[at] = v;
    else if (t0 + r < T && e0 + e < E)
      logits[(size_t)(t0 + r) * E + e0 + e] = v;
  }
  if (parts == 1) return;
  cluster.sync();
  for (int o = part * 256 + tid; o < kRt * kRe; o += parts * 256) {
    const int r = o / kRe, e = o - r * kRe, at = r * kRo + e;
    float v = *cluster.map_shared_rank(sums + at, 0);
    for (int q = 1; q < parts; ++q) v += *cluster.map_shared_rank(sums + at, q);
    if (t0 + r < T && e0 + e < E) logits[(size_t)(t0 + r) * E + e0 + e] = v;
  }
  cluster.sync();      // the last sums have been read
}

template <int V>
static int launch_router_tiles(const bf16* x, const float* rw, int H, int E, int T, int sms, float* logits, cudaStream_t stream) {
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard g{once}; g.needed()) {
    if (cudaFuncSetAttribute(router_logits_tile_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRouterSmem) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    g.done();
  }
  const int et = (E + kRe - 1) / kRe, tt = (T + kRt - 1) / kRt, steps = (H + kRk - 1) / kRk;
  // A block alone keeps its SM as busy as two do, so the time is that of the fullest SM: blocks of it x (steps of a block + what a block
  // costs besides, 2.5 steps). 256 experts of 3072, tiles with 1 / 2 / 4 / 8 parts, us (all measured with a form
  // 10 % slower): 96 tiles 108 / 106 / 83 / 92, 64 tiles 107 / 60 / 57 / 64,
  // 32 tiles 106 / 58 / 33 / 32, 256 tiles 200 / 204 / 208 / 219.
  int parts = 1;
  double best = 0.;
  for (int c = 1; c <= 8 && c <= steps; c *= 2) {
    const double cost = (double)(((long long)et * tt * c + sms - 1) / sms) * ((steps + c - 1) / c + 2.5);
    if (c == 1 || cost < best) {
      best = cost;
      parts = c;
    }
  }
  pk_prefer_max_smem((const void*)router_logits_tile_kernel<V>);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(parts, et, tt);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = kRouterSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pk_pdl_enabled() ? 2 : 1;
  if (const cudaError_t e = cudaLaunchKernelEx(&cfg, router_logits_tile_kernel<V>, x, rw, H, E, T, logits); e != cudaSuccess) {
    pk_set_last_cuda_error((int)e);
    return PK_ERR_CUDA;
  }
  return PK_OK;
}

// One block per token: scores from the logits, top-k with lowest-id tie break.
// score_func 0 softmax, 1 sigmoid, 2 sqrt(softplus); selection on score + bias.
__global__ void __launch_bounds__(256) router_topk_kernel(const float* logits, const float* bias, int E,
                                                          int topk, int score_func, int norm_topk, float route_scale,
                                                          int* ids, float* weights) {
  pk::pdl_wait();
  pk::pdl_trigger_few();      // routing the same tokens again and again: 592 by 8 experts of 1024 13.2 -> 11.2 us, 1000 by 256 of 3072 95 -> 57
  extern __shared__ float sm[];  // [E] scores, [E] selection keys
  float* sc = sm;
  float* key = sc + E;
  __shared__ float red[40];
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < E; e += 256) sc[e] = logits[(size_t)t * E + e];
  __syncthreads();
  if (score_func == 0) {
    float mx = -INFINITY;
    for (int e = tid; e < E; e += 256) mx = fmaxf(mx, sc[e]);
    mx = block_max(mx, red);
    float s = 0.f;
    for (int e = tid; e < E; e += 256) {
      sc[e] = __expf(sc[e] - mx);
      s += sc[e];
    }
    s = block_sum(s, red);
    for (int e = tid; e < E; e += 256) sc[e] /= s;
  } else {
    for (int e = tid; e < E; e += 256) sc[e] = score_func == 1 ? sigmoidf_(sc[e]) : sqrtf(softplusf_(sc[e]));
  }
  __syncthreads();
  // keys stay finite: a NaN or -inf key would never win a comparison below, the pick would keep its initial invalid id
  // and index shared memory with it
  for (int e = tid; e < E; e += 256) {
    const float k = sc[e] + (bias ? bias[e] : 0.f);
    key[e] = k > -3.0e38f ? k : -3.0e38f;
  }
  __syncthreads();
  if (warp == 0) {
    float wsum = 0.f;
    for (int j = 0; j < topk; ++j) {
      float bv = -INFINITY;
      int bi = 0x7fffffff;
      for (int e = lane; e < E; e += 32)
        if (key[e] > bv) { bv = key[e]; bi = e; }
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (lane == 0) {
        ids[(size_t)t * topk + j] = bi;
        weights[(size_t)t * topk + j] = sc[bi];
        key[bi] = -INFINITY;
      }
      wsum += sc[bi];
      __syncwarp();
    }
    if (lane < topk) {
      float w = weights[(size_t)t * topk + lane];
      if (norm_topk) w /= (wsum > 0.f ? wsum : 1.f);
      weights[(size_t)t * topk + lane] = w * route_scale;
    }
  }
}

// Group routes by expert, those of an expert in increasing route index (one block). Every warp counts a contiguous share of the
// routes in counters of its own, the counts become offsets (warp by warp within an expert, expert by expert), and the warps walk
// their shares again: 32 routes at a time, a route's place among them from a match of the expert ids. The first form scanned all
// routes once per expert: 238 us for 4096 routes over 256 experts, against 11 us.
__global__ void __launch_bounds__(1024) group_routes_kernel(const int* ids, const float* weights, int T, int topk, int E,
                                                            int* seg_start, int* route_token, float* route_weight,
                                                            int* route_src) {
  pk::pdl_wait();
  pk::pdl_trigger();
  extern __shared__ int cnt[];  // [warps][E]
  __shared__ int part[33];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5, R = T * topk;
  const int share = ((R + warps - 1) / warps + 31) & ~31, r0 = min(warp * share, R), r1 = min(r0 + share, R);
  for (int e = tid; e < warps * E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  int* mine = cnt + warp * E;
  for (int r = r0 + lane; r < r1; r += 32) {
    const int e = ids[r];
    if ((unsigned)e < (unsigned)E) atomicAdd(&mine[e], 1);
#if PK_DEBUG_BUILD
    else PK_DEBUG_RECORD(102, e, E);
#endif
  }
  __syncthreads();
  // counts of a block of experts -> offsets; `run` routes before the block
  int run = 0;
  for (int e0 = 0; e0 < E; e0 += blockDim.x) {
    const int e = e0 + tid;
    int n = 0;
    if (e < E)
      for (int w = 0; w < warps; ++w) {
        const int c = cnt[w * E + e];
        cnt[w * E + e] = n;
        n += c;
      }
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    int before = run;
    for (int w = 0; w < warp; ++w) before += part[w];
    int total = 0;
    for (int w = 0; w < warps; ++w) total += part[w];
    if (e < E) {
      const int start = before + inc - n;
      seg_start[e] = start;
      for (int w = 0; w < warps; ++w) cnt[w * E + e] += start;
    }
    run += total;
    __syncthreads();
  }
  if (tid == 0) seg_start[E] = run;
  for (int base = r0; base < r1; base += 32) {
    const int r = base + lane, e = r < r1 ? ids[r] : -1;
    const bool ok = (unsigned)e < (unsigned)E;
    const unsigned same = __match_any_sync(0xffffffffu, ok ? e : -1);
    const int rank = __popc(same & ((1u << lane) - 1u));
    const int pos = ok ? mine[e] + rank : 0;
    __syncwarp();
    if (ok) {
      if (rank == 0) mine[e] += __popc(same);
      route_token[pos] = r / topk;
      route_weight[pos] = weights[r];
      if (route_src) route_src[pos] = r;
    }
    __syncwarp();
  }
}

// Quantised embedding: decode selected rows to bf16 (one warp per 256 weights).
__global__ void __launch_bounds__(256) gguf_dequant_rows_kernel(const uint8_t* W, int type, const int* rows, int nrows,
                                                                int K, int row_offset, int table_rows, bf16* out) {
  pk::pdl_wait();
  pk::pdl_trigger();
  // one warp per 256-weight block, walking (row, block) units with a grid stride; a lane's eight weights leave as one
  // 16-byte store
  const int lane = threadIdx.x & 31;
  const int nblk = K >> 8;
  const size_t rb = row_bytes(type, K);
  const long long units = (long long)nrows * nblk;
  for (long long u = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += (long long)gridDim.x * 8) {
    const int r = (int)(u / nblk), blk = (int)(u - (long long)r * nblk);
    const int src = (rows ? rows[r] : r) - row_offset;
    const bool mine = src >= 0 && src < table_rows;
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = 0.f;
    if (mine) {
      const uint8_t* b = W + (size_t)src * rb + (size_t)blk * block_bytes(type);
      switch (type) {
        case T_IQ2_XXS: decode8<T_IQ2_XXS>(b, lane, w); break;
        case T_Q2_K: decode8<T_Q2_K>(b, lane, w); break;
        case T_IQ1_M: decode8<T_IQ1_M>(b, lane, w); break;
        case T_Q4_K: decode8<T_Q4_K>(b, lane, w); break;
        case T_Q5_K: decode8<T_Q5_K>(b, lane, w); break;
        case T_IQ2_XS: decode8<T_IQ2_XS>(b, lane, w); break;
        case T_IQ3_XXS: decode8<T_IQ3_XXS>(b, lane, w); break;
        case T_IQ4_XS: decode8<T_IQ4_XS>(b, lane, w); break;
        case T_Q6_K: decode8<T_Q6_K>(b, lane, w); break;
        case T_Q8_0: decode8<T_Q8_0>(b, lane, w); break;
        case T_MXFP4: decode8<T_MXFP4>(b, lane, w); break;
        default: decode8<T_BF16>(b, lane, w); break;
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 pr = __floats2bfloat162_rn(w[2 * i], w[2 * i + 1]);
      o[i] = *reinterpret_cast<const uint32_t*>(&pr);
    }
    *reinterpret_cast<uint4*>(out + (size_t)r * K + (blk << 8) + (lane << 3)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int M>
int launch_linear(const LinearParams& p_in, int sm_count, cudaStream_t stream) {
  LinearParams p = p_in;
  p.stage_bytes = M <= 2 ? stage_bytes_per_warp(p.type, p.K) : 0;
  const size_t smem = (size_t)M * p.K * sizeof(float) + (size_t)kWarps * p.stage_bytes;
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(gguf_linear_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 184 * 1024) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  const int groups = p.epi == 1 ? p.N / 2 : p.N;
  int blocks = (groups + kWarps - 1) / kWarps;
  blocks = min(blocks, (sm_count > 0 ? sm_count : 148) * 8);
  gguf_linear_kernel<M><<<blocks, kThreads, smem, stream>>>(p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

}  // namespace

PK_API int pk_gguf_block_bytes(int type) { return (type >= 0 && type <= T_LAST) ? block_bytes(type) : 0; }

// x bf16 [M, K] (M <= 8, M * K * 4 bytes <= 200 KB), W raw rows, K a multiple of 256.
PK_API int pk_gguf_linear(const void* W, int type, int N, int K, int M, const void* x, const float* gamma, float eps,
                          int epi, void* y, int ldy, int sm_count, cudaStream_t stream) {
  if (type < 0 || type > T_LAST || M < 1 || M > 8 || (K & 255) != 0 || N < 1) return PK_ERR_BAD_ARG;
  if ((size_t)M * K * 4 > 184 * 1024) return PK_ERR_UNSUPPORTED;   // plus the warps' stage buffers
  if (epi == 1 && (N & 1)) return PK_ERR_BAD_ARG;
  LinearParams p{(const uint8_t*)W, type, N, K, M, (const pk::bf16*)x, gamma, eps, epi, y, ldy, 0};
  switch (M) {
    case 1: return launch_linear<1>(p, sm_count, stream);
    case 2: return launch_linear<2>(p, sm_count, stream);
    case 3: case 4: p.M = M; return launch_linear<4>(p, sm_count, stream);
    default: return launch_linear<8>(p, sm_count, stream);
  }
}

// Per-device scratch for the router logits [T, E]; grows on demand (a growth inside a stream capture fails: run one
// step of the same size before capturing, which callers do anyway to warm the kernels up).
static float* router_scratch(size_t floats) {
  static float* buf[64] = {};
  static size_t cap[64] = {};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (cap[dev] < floats) {
    float* nb = nullptr;
    const size_t want = floats < 4096 ? 4096 : floats;
    if (cudaMalloc((void**)&nb, want * sizeof(float)) != cudaSuccess) return nullptr;
    // the old buffer may still be in use by kernels in flight: it is left to the process lifetime (sizes settle quickly)
    buf[dev] = nb;
    cap[dev] = want;
  }
  return buf[dev];
}

// The blocks of the form with one warp per expert keep up to eight tokens of H floats each in shared memory; when they are more than are
// resident at once, the tiles are faster, if an expert tile is full. One warp per expert / tiles, us: 256 experts of 3072 (256 blocks for
// 64 tokens, 296 resident), 64 tokens 15 / 17, 96 tokens 28 / 17, 256 tokens 56 / 27; 128 of 4096 (148 resident), 64 tokens 13 / 21, 96 tokens
// 27 / 21, 512 tokens 86 / 34; 64 of 2048 (444 resident), 384 tokens 13 / 13, 512 tokens 26 / 13;
// one token by 256 experts of 8192 9 / 39.
static bool router_tiles(int T, int E, int H, int sms) {
  const long long resident = std::max(1, std::min(8, (227 * 1024) / (4 * std::min(T, 8) * H + 1024)));
  return E >= kRe && (long long)((E + 7) / 8) * ((T + 7) / 8) > resident * sms;
}

PK_API int pk_router_topk(const void* x, const float* router_w, const float* bias, int T, int H, int E, int topk,
                          int score_func, int norm_topk, float route_scale, int* ids, float* weights,
                          cudaStream_t stream) {
  if (T < 1 || topk < 1 || topk > 32 || topk > E) return PK_ERR_BAD_ARG;
  const int tile = T < 8 ? T : 8;
  const size_t smem_x = (size_t)tile * H * sizeof(float);
  if (smem_x > 200 * 1024 || (size_t)2 * E * sizeof(float) > 48 * 1024) return PK_ERR_UNSUPPORTED;
  if (smem_x > 48 * 1024) {
    static PkDeviceOnce once;
    if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
      if (cudaFuncSetAttribute(router_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) {
        pk_set_last_cuda_error((int)cudaGetLastError());
        return PK_ERR_CUDA;
      }
      once_guard.done();
    }
  }
  float* logits = router_scratch((size_t)T * E);
  if (logits == nullptr) return PK_ERR_CUDA;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return PK_ERR_CUDA;
  if (router_tiles(T, E, H, sms)) {
    const bool by16 = (H & 7) == 0 && (((uintptr_t)x | (uintptr_t)router_w) & 15) == 0, by4 = (H & 1) == 0 && ((uintptr_t)x & 3) == 0;
    const auto launch = by16 ? launch_router_tiles<8> : by4 ? launch_router_tiles<2> : launch_router_tiles<1>;
    if (const int rc = launch((const pk::bf16*)x, router_w, H, E, T, sms, logits, stream)) return rc;
  } else
    PK_LAUNCH_PDL(router_logits_kernel, dim3((E + 7) / 8, (T + 7) / 8), dim3(256), smem_x, stream, (const pk::bf16*)x, router_w, H, E, T, logits);
  PK_CHECK_LAUNCH();
  PK_LAUNCH_PDL(router_topk_kernel, dim3(T), dim3(256), (size_t)2 * E * sizeof(float), stream, logits, bias, E, topk, score_func, norm_topk, route_scale, ids,
                                                                        weights);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_group_routes(const int* ids, const float* weights, int T, int topk, int E, int* seg_start, int* route_token,
                           float* route_weight, int* route_src, cudaStream_t stream) {
  if (E + 1 > 12000) return PK_ERR_UNSUPPORTED;
  const int R = T * topk;
  // warps for the routes and, with few of them, for the walk over the experts: one token of 256 / 2000 experts 5.0 / 27.7 -> 3.4 / 8.5 us
  int warps = min(32, max((E + 63) / 64, (R + 31) / 32));
  while (warps > 4 && (size_t)warps * E * sizeof(int) > 192 * 1024) warps >>= 1;
  const size_t smem = (size_t)warps * E * sizeof(int);
  if (smem > kPlainSmem) {
    static PkDeviceOnce once;
    if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
      if (cudaFuncSetAttribute(group_routes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 192 * 1024) != cudaSuccess) {
        pk_set_last_cuda_error((int)cudaGetLastError());
        return PK_ERR_CUDA;
      }
      once_guard.done();
    }
  }
  PK_LAUNCH_PDL_L1(group_routes_kernel, dim3(1), dim3(warps * 32), smem, stream, ids, weights, T, topk, E, seg_start, route_token, route_weight, route_src);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// Routed experts of one rank: experts [expert_offset, expert_offset + local_experts) live in
// W13 / W2. y (fp32 [T, H]) must be zeroed by the caller; hbuf holds R * I floats.
// y[t] += sum over the token's routes (in route order) of route_weight * ybuf[route]; routes of experts outside
// [expert_offset, expert_offset + local_experts) are skipped. route_pos: int scratch [T * topk].
PK_API int pk_moe_reduce_routes(const float* ybuf, const float* route_weight, const int* route_src, const int* seg_start, int T, int topk, int H,
                                int expert_offset, int local_experts, int* route_pos, float* y, cudaStream_t stream) {
  if (ybuf == nullptr || route_weight == nullptr || route_src == nullptr || seg_start == nullptr || route_pos == nullptr || y == nullptr || T < 1 || topk < 1)
    return PK_ERR_BAD_ARG;
  const int R = T * topk;
  PK_LAUNCH_PDL(invert_routes_kernel, dim3((R + 255) / 256), dim3(256), 0, stream, route_src, R, route_pos);
  PK_CHECK_LAUNCH();
  PK_LAUNCH_PDL_L1(moe_reduce_routes_weighted_kernel, dim3((H + 255) / 256, T), dim3(256), 0, stream, ybuf, route_weight, route_pos, seg_start, topk, H, expert_offset,
                                                                                  local_experts, y);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// route_pos[route_src[pos]] = pos: where route (t, k) sits in the expert-sorted order.
PK_API int pk_invert_routes(const int* route_src, int R, int* route_pos, cudaStream_t stream) {
  if (route_src == nullptr || route_pos == nullptr || R < 1) return PK_ERR_BAD_ARG;
  PK_LAUNCH_PDL(invert_routes_kernel, dim3((R + 255) / 256), dim3(256), 0, stream, route_src, R, route_pos);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

static int moe_forward_impl(const void* W13, const void* W2, int type13, int type2, int E, int H, int I, const void* x,
                            const int* seg_start, const int* route_token, const float* route_weight, float* hbuf, float* y,
                            float limit, int expert_offset, int local_experts, int sm_count, float* ybuf, cudaStream_t stream,
                            int total_routes = 0);

PK_API int pk_gguf_moe_forward(const void* W13, const void* W2, int type13, int type2, int E, int H, int I,
                               const void* x, const int* seg_start, const int* route_token, const float* route_weight,
                               float* hbuf, float* y, float limit, int expert_offset, int local_experts, int sm_count,
                               cudaStream_t stream) {
  return moe_forward_impl(W13, W2, type13, type2, E, H, I, x, seg_start, route_token, route_weight, hbuf, y, limit, expert_offset,
                          local_experts, sm_count, nullptr, stream);
}

// Same result up to rounding, but bitwise reproducible: every route writes its own output row (ybuf, R * H
// floats) and a second kernel adds the rows of each token in route order. route_src comes from pk_group_routes;
// route_pos is R ints of scratch; T tokens with topk routes each.
PK_API int pk_gguf_moe_forward_det(const void* W13, const void* W2, int type13, int type2, int E, int H, int I, const void* x,
                                   const int* seg_start, const int* route_token, const float* route_weight, const int* route_src,
                                   float* hbuf, float* ybuf, int* route_pos, float* y, int T, int topk, float limit,
                                   int expert_offset, int local_experts, int sm_count, cudaStream_t stream) {
  if (route_src == nullptr || ybuf == nullptr || route_pos == nullptr || T < 1 || topk < 1) return PK_ERR_BAD_ARG;
  const int R = T * topk;
  const int rc = moe_forward_impl(W13, W2, type13, type2, E, H, I, x, seg_start, route_token, route_weight, hbuf, y, limit,
                                  expert_offset, local_experts, sm_count, ybuf, stream, R);
  if (rc != PK_OK) return rc;
  PK_LAUNCH_PDL(invert_routes_kernel, dim3((R + 255) / 256), dim3(256), 0, stream, route_src, R, route_pos);
  PK_CHECK_LAUNCH();
  moe_reduce_routes_kernel<<<dim3((H + 255) / 256, T), 256, 0, stream>>>(ybuf, route_pos, seg_start, topk, H, expert_offset,
                                                                         local_experts, y);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

static int moe_forward_impl(const void* W13, const void* W2, int type13, int type2, int E, int H, int I, const void* x,
                            const int* seg_start, const int* route_token, const float* route_weight, float* hbuf, float* y,
                            float limit, int expert_offset, int local_experts, int sm_count, float* ybuf, cudaStream_t stream,
                            int total_routes) {
  if ((H & 255) || (I & 255) || local_experts < 1) return PK_ERR_BAD_ARG;
  if ((size_t)8 * H * 4 > 184 * 1024 || (size_t)8 * I * 4 > 184 * 1024) return PK_ERR_UNSUPPORTED;   // plus the warps' stage buffers
  MoeParams p{(const uint8_t*)W13, (const uint8_t*)W2, type13, type2, E, H, I, (const pk::bf16*)x, seg_start, route_token,
              route_weight, hbuf, y, limit, expert_offset, local_experts, ybuf};
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(gguf_moe_w13_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 184 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(gguf_moe_w2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 184 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(gguf_moe_w13_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 184 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(gguf_moe_w2_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 184 * 1024) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  (void)sm_count;
  if (total_routes > 0 && total_routes <= kRouteParallelMax) {
    // one block set per route: at most total_routes of them belong to this rank
    MoeParams q = p;
    const int t13 = (I + kWarps - 1) / kWarps, t2 = (H + kWarps - 1) / kWarps;
    gguf_moe_w13_route_kernel<<<dim3(t13 < 256 ? t13 : 256, total_routes), kThreads,
                                (size_t)H * 4 + (size_t)kWarps * stage_bytes_per_warp(type13, H), stream>>>(q);
    PK_CHECK_LAUNCH();
    gguf_moe_w2_route_kernel<<<dim3(t2 < 256 ? t2 : 256, total_routes), kThreads,
                               (size_t)I * 4 + (size_t)kWarps * stage_bytes_per_warp(type2, I), stream>>>(q);
    PK_CHECK_LAUNCH();
    return PK_OK;
  }
  const int tiles13 = min((I + kWarps - 1) / kWarps, 32), tiles2 = min((H + kWarps - 1) / kWarps, 32);
  gguf_moe_w13_kernel<<<dim3(tiles13, local_experts), kThreads, (size_t)8 * H * 4, stream>>>(p);
  PK_CHECK_LAUNCH();
  gguf_moe_w2_kernel<<<dim3(tiles2, local_experts), kThreads, (size_t)8 * I * 4, stream>>>(p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// out[r, :] = dequant(W[rows[r] - row_offset, :]) as bf16; rows outside the local table give zeros
// (vocabulary-sharded embedding). rows == null means rows 0..nrows-1.
PK_API int pk_gguf_dequant_rows(const void* W, int type, const int* rows, int nrows, int K, int row_offset,
                                int table_rows, void* out, cudaStream_t stream) {
  if (type < 0 || type > T_LAST || (K & 255) != 0 || nrows < 1) return PK_ERR_BAD_ARG;
  if (((uintptr_t)out & 15) != 0) return PK_ERR_BAD_ARG;
  const long long units = (long long)nrows * (K >> 8);
  const long long want = (units + 7) / 8;
  const int grid = (int)(want < 148LL * 32 ? want : 148LL * 32);
  PK_LAUNCH_PDL_L1(gguf_dequant_rows_kernel, dim3(grid), dim3(256), 0, stream, (const uint8_t*)W, type, rows, nrows, K, row_offset, table_rows,
                                                    (pk::bf16*)out);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
