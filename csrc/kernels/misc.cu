// Small memory-bound ops: embedding gather, RMSNorm with fused residual/reduce-in,
// SwiGLU, argmax / top-k candidates over fp32 logits, epoch bump for the comm protocol.
// Reference counterparts: cpp_engine/cuda/qwen_half_ops.cu:693-709 (rmsnorm, (1+gamma)),
// 1529 (embedding), cpp_engine/cuda/cuda_ops.cu:40-128 (argmax_fp32, argmax_fp32_rows).
#include <cuda_fp8.h>

#include "../common/pk_comm.cuh"
#include "../common/pk_common.cuh"

namespace {

using namespace pk;

// Vocabulary-sharded gather: rows outside [vocab_start, vocab_start + rows) give zeros,
// so that the sum over ranks is the embedding.
__global__ void embedding_kernel(const int* tokens, const bf16* table, int dim, int vocab_start,
                                 int vocab_rows, bf16* out_bf16, float* out_f32) {
  const int m = blockIdx.x;
  const int tok = tokens[m] - vocab_start;
  const bool mine = tok >= 0 && tok < vocab_rows;
  if (out_f32 == nullptr && out_bf16 != nullptr && (dim & 7) == 0 && (((uintptr_t)table | (uintptr_t)out_bf16) & 15) == 0) {
    // 16 bytes at a time: 512 rows of 5120 took 12 us by two bytes, now 4
    const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)(mine ? tok : 0) * dim);
    uint4* dst = reinterpret_cast<uint4*>(out_bf16 + (size_t)m * dim);
    for (int k = threadIdx.x; k < dim >> 3; k += blockDim.x) dst[k] = mine ? __ldg(src + k) : make_uint4(0, 0, 0, 0);
    return;
  }
  for (int k = threadIdx.x; k < dim; k += blockDim.x) {
    const bf16 v = mine ? table[(size_t)tok * dim + k] : __float2bfloat16(0.f);
    if (out_bf16) out_bf16[(size_t)m * dim + k] = v;
    if (out_f32) out_f32[(size_t)m * dim + k] = __bfloat162float(v);
  }
}

struct NormParams {
  const bf16* x;       // [M, K] or null
  const float* parts;  // [nparts, M, K] or null
  int nparts;
  int M, K;
  bf16* hidden_out;    // x + sum(parts), bf16 (may be null)
  const float* gamma;
  int mode;            // 1: (1+gamma), 2: gamma
  float eps;
  bf16* y;             // [M, K]
  PkWait wait;
};

__global__ void __launch_bounds__(256) rmsnorm_kernel(const NormParams p) {
  pk::pdl_wait();
  pk::pdl_trigger_few();
  extern __shared__ float row[];
  __shared__ float red[40];
  const int m = blockIdx.x;
  if (p.parts != nullptr && p.wait.flag != nullptr) {
    if (threadIdx.x == 0) wait_all_ranks(p.wait);
    __syncthreads();
  }
  float ss = 0.f;
  for (int k = threadIdx.x; k < p.K; k += blockDim.x) {
    const size_t gi = (size_t)m * p.K + k;
    float v = p.x ? __bfloat162float(p.x[gi]) : 0.f;
    for (int r = 0; r < p.nparts; ++r) v += p.parts[((size_t)r * p.M + m) * p.K + k];
    const bf16 hv = __float2bfloat16(v);
    if (p.hidden_out) p.hidden_out[gi] = hv;
    v = __bfloat162float(hv);
    row[k] = v;
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float r = rsqrtf(ss / (float)p.K + p.eps);
  if (p.y == nullptr) return;
  for (int k = threadIdx.x; k < p.K; k += blockDim.x) {
    const float g = p.gamma[k];
    p.y[(size_t)m * p.K + k] = __float2bfloat16(row[k] * r * (p.mode == 1 ? 1.f + g : g));
  }
}

// The same for rows of whole 16-byte pieces (K a multiple of 8, aligned): a thread has eight neighbouring elements at a time and all
// its loads of an iteration under way together. One row of 3072: 9.3 -> 3.3 us, 1500 rows 23 -> 13 us (the form above loads
// two bytes, waits and goes on).
__global__ void __launch_bounds__(256) rmsnorm_vec_kernel(const NormParams p) {
  pk::pdl_wait();
  pk::pdl_trigger_few();
  extern __shared__ __align__(16) float row[];
  __shared__ float red[40];
  const size_t base = (size_t)blockIdx.x * p.K;
  if (p.parts != nullptr && p.wait.flag != nullptr) {
    if (threadIdx.x == 0) wait_all_ranks(p.wait);
    __syncthreads();
  }
  float ss = 0.f;
#pragma unroll 2
  for (int k = threadIdx.x * 8; k < p.K; k += 2048) {
    const uint4 raw = p.x ? *reinterpret_cast<const uint4*>(p.x + base + k) : make_uint4(0, 0, 0, 0);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __uint_as_float(w[j] << 16);
      v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
    for (int r = 0; r < p.nparts; ++r) {
      const float4* q = reinterpret_cast<const float4*>(p.parts + (size_t)r * p.M * p.K + base + k);
      const float4 a = q[0], b = q[1];
      v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
      v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
    }
    uint32_t h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 pr = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      h[j] = *reinterpret_cast<const uint32_t*>(&pr);
      v[2 * j] = __uint_as_float(h[j] << 16);
      v[2 * j + 1] = __uint_as_float(h[j] & 0xffff0000u);
    }
    if (p.hidden_out) *reinterpret_cast<uint4*>(p.hidden_out + base + k) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(row + k) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(row + k + 4) = make_float4(v[4], v[5], v[6], v[7]);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
  }
  ss = block_sum(ss, red);
  if (p.y == nullptr) return;
  const float r = rsqrtf(ss / (float)p.K + p.eps), one = p.mode == 1 ? 1.f : 0.f;
#pragma unroll 2
  for (int k = threadIdx.x * 8; k < p.K; k += 2048) {
    const float4 g0 = __ldg(reinterpret_cast<const float4*>(p.gamma + k)), g1 = __ldg(reinterpret_cast<const float4*>(p.gamma + k + 4));
    const float4 a = *reinterpret_cast<const float4*>(row + k), b = *reinterpret_cast<const float4*>(row + k + 4);
    const __nv_bfloat162 o0 = __floats2bfloat162_rn(a.x * r * (one + g0.x), a.y * r * (one + g0.y)), o1 = __floats2bfloat162_rn(a.z * r * (one + g0.z), a.w * r * (one + g0.w));
    const __nv_bfloat162 o2 = __floats2bfloat162_rn(b.x * r * (one + g1.x), b.y * r * (one + g1.y)), o3 = __floats2bfloat162_rn(b.z * r * (one + g1.z), b.w * r * (one + g1.w));
    *reinterpret_cast<uint4*>(p.y + base + k) = make_uint4(*reinterpret_cast<const uint32_t*>(&o0), *reinterpret_cast<const uint32_t*>(&o1),
                                                            *reinterpret_cast<const uint32_t*>(&o2), *reinterpret_cast<const uint32_t*>(&o3));
  }
}

// RMSNorm of bf16 rows with 16-byte accesses, optionally followed in the same kernel by the activation quantisation
// of the native FP8 GEMM (the layout and arithmetic of quant_act_fp8_kernel in gemm_fp8.cu, on the bf16-rounded
// outputs: one scale per row and 128-wide k block = amax / 448, the E4M3 code of y / scale and, with two terms, the code
// of the rounding residue). Sixteen consecutive threads hold one k block, so its amax is four shuffles.
struct NormQuantParams {
  const bf16* x;   // [M, K]
  int M, K;
  const float* gamma;
  int mode;        // 1: (1+gamma), 2: gamma
  float eps;
  bf16* y;         // [M, K]
  int terms;       // 0: no quantisation
  uint8_t* q;      // [terms][m_pad][K]
  int m_pad;
  float* scale_t;  // [K / 128][s_ld]
  int s_ld;
};

__global__ void __launch_bounds__(256) rmsnorm_quant_kernel(const NormQuantParams p) {
  pk::pdl_wait();
  pk::pdl_trigger();
  extern __shared__ __align__(16) float row[];
  __shared__ float red[40];
  const int m = blockIdx.x, tid = threadIdx.x, nvec = p.K >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(p.x + (size_t)m * p.K);
  float ss = 0.f;
  for (int v = tid; v < nvec; v += 256) {
    const uint4 raw = xr[v];
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      row[v * 8 + 2 * j] = a;
      row[v * 8 + 2 * j + 1] = b;
      ss += a * a + b * b;
    }
  }
  ss = block_sum(ss, red);
  const float r = rsqrtf(ss / (float)p.K + p.eps);
  // every thread runs every iteration: the shuffles below need whole warps
  for (int v0 = 0; v0 < nvec; v0 += 256) {
    const int v = v0 + tid;
    const bool on = v < nvec;
    float yv[8];
    uint32_t packed[4] = {0u, 0u, 0u, 0u};
    float amax = 0.f;
    if (on) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float g = p.gamma[v * 8 + j];
        const bf16 h = __float2bfloat16(row[v * 8 + j] * r * (p.mode == 1 ? 1.f + g : g));
        yv[j] = __bfloat162float(h);
        amax = fmaxf(amax, fabsf(yv[j]));
        packed[j >> 1] |= (uint32_t)__bfloat16_as_ushort(h) << (16 * (j & 1));
      }
      *reinterpret_cast<uint4*>(p.y + (size_t)m * p.K + v * 8) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
    if (p.terms > 0) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      if (on) {
        const float s = amax > 0.f ? amax * (1.f / 448.f) : 1.f;
        const float inv = 1.f / s;
        uint32_t hi[2] = {0u, 0u}, lo[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float t = yv[j] * inv;
          const __nv_fp8_storage_t c = __nv_cvt_float_to_fp8(t, __NV_SATFINITE, __NV_E4M3);
          hi[j >> 2] |= (uint32_t)c << (8 * (j & 3));
          const float back = __half2float(__half(__nv_cvt_fp8_to_halfraw(c, __NV_E4M3)));
          lo[j >> 2] |= (uint32_t)__nv_cvt_float_to_fp8(t - back, __NV_SATFINITE, __NV_E4M3) << (8 * (j & 3));
        }
        const size_t off = (size_t)m * p.K + v * 8;
        *reinterpret_cast<uint2*>(p.q + off) = make_uint2(hi[0], hi[1]);
        if (p.terms > 1) *reinterpret_cast<uint2*>(p.q + (size_t)p.m_pad * p.K + off) = make_uint2(lo[0], lo[1]);
        if ((tid & 15) == 0) p.scale_t[(size_t)(v >> 4) * p.s_ld + m] = s;
      }
    }
  }
}

// Reduce-scatter / all-gather form of the tensor-parallel RMSNorm (prefill): this rank owns rows
// [rank * rpr, rank * rpr + rows_mine). For each of them: x = hidden + sum_r parts[r] (fp32 partial rows that the
// row-parallel GEMM epilogues of every rank pushed here), hidden = bf16(x) (kept on the owner only), y = rmsnorm(x),
// and y is stored as bf16 into EVERY rank's copy of the normalised activations (the all-gather, fused into the norm).
// Then the rank publishes its all-gather flag and waits for the others', so that the kernel's end means "all rows of y
// are here". Per site a rank sends (world-1)/world of one fp32 row block plus (world-1) bf16 row blocks instead of
// world fp32 copies of everything.
struct NormAgParams {
  bf16* hidden;          // local [M, K] residual stream; only the owned rows are read and written
  const float* parts;    // local slot [world][rpr][K] fp32
  int world, rank, rpr, rows_mine, K;
  const float* gamma;
  int mode;
  float eps;
  bf16* y_peer[PK_MAX_RANKS];      // every rank's [M, K] bf16 buffer of normalised rows (own one included)
  PkWait wait_rs;        // flags of the reduce-scatter pushes (all ranks have stored their partials)
  PkPush pub_ag;         // flags of the all-gather (dst unused)
  PkWait wait_ag;
};

__global__ void __launch_bounds__(256) rmsnorm_rs_ag_kernel(const NormAgParams p) {
  extern __shared__ float row[];
  __shared__ float red[40];
  if (threadIdx.x == 0) wait_all_ranks(p.wait_rs);
  __syncthreads();
  for (int ml = blockIdx.x; ml < p.rows_mine; ml += gridDim.x) {
    const int m = p.rank * p.rpr + ml;
    float ss = 0.f;
    for (int k = threadIdx.x; k < p.K; k += blockDim.x) {
      float v = __bfloat162float(p.hidden[(size_t)m * p.K + k]);
      for (int r = 0; r < p.world; ++r) v += p.parts[((size_t)r * p.rpr + ml) * p.K + k];
      const bf16 hv = __float2bfloat16(v);
      p.hidden[(size_t)m * p.K + k] = hv;
      v = __bfloat162float(hv);
      row[k] = v;
      ss += v * v;
    }
    ss = block_sum(ss, red);
    const float rs = rsqrtf(ss / (float)p.K + p.eps);
    for (int k2 = threadIdx.x * 2; k2 < p.K; k2 += blockDim.x * 2) {
      const float g0 = p.gamma[k2], g1 = p.gamma[k2 + 1];
      const __nv_bfloat162 yv = __floats2bfloat162_rn(row[k2] * rs * (p.mode == 1 ? 1.f + g0 : g0),
                                                      row[k2 + 1] * rs * (p.mode == 1 ? 1.f + g1 : g1));
      for (int r = 0; r < p.world; ++r) *reinterpret_cast<__nv_bfloat162*>(p.y_peer[r] + (size_t)m * p.K + k2) = yv;
    }
    __syncthreads();   // `row` is reused by the block's next row
  }
  publish_when_grid_done(p.pub_ag);
  if (threadIdx.x == 0) wait_all_ranks(p.wait_ag);
}

__global__ void silu_mul_kernel(const bf16* gu, int inter, bf16* out, float limit) {
  // gu: [M, 2*inter] = gate | up
  const int m = blockIdx.y;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= inter) return;
  float g = __bfloat162float(gu[(size_t)m * 2 * inter + j]);
  float u = __bfloat162float(gu[(size_t)m * 2 * inter + inter + j]);
  if (limit > 0.f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
  }
  out[(size_t)m * inter + j] = __float2bfloat16(silu(g) * u);
}

// Stage 1 of a row argmax: each block scans a slice and keeps (value, index) with the
// lowest index on ties. Stage 2 merges the slices. Output candidate = {logit, token id}.
__global__ void __launch_bounds__(256) argmax_stage1(const float* logits, int ld, int n, int id_offset,
                                                     float* cand_val, int* cand_idx) {
  const int m = blockIdx.y, nb = gridDim.x;
  const int per = (n + nb - 1) / nb;
  const int lo = blockIdx.x * per, hi = min(n, lo + per);
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const float v = logits[(size_t)m * ld + i];
    if (v > best || (v == best && i < bi)) {
      best = v;
      bi = i;
    }
  }
  __shared__ float sv[256];
  __shared__ int si[256];
  sv[threadIdx.x] = best;
  si[threadIdx.x] = bi;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      const float ov = sv[threadIdx.x + s];
      const int oi = si[threadIdx.x + s];
      if (ov > sv[threadIdx.x] || (ov == sv[threadIdx.x] && oi < si[threadIdx.x])) {
        sv[threadIdx.x] = ov;
        si[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    cand_val[m * nb + blockIdx.x] = sv[0];
    cand_idx[m * nb + blockIdx.x] = si[0] == 0x7fffffff ? 0x7fffffff : si[0] + id_offset;
  }
}

__global__ void argmax_stage2(const float* cand_val, const int* cand_idx, int ncand, float* out_val,
                              int* out_idx) {
  const int m = blockIdx.x;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < ncand; i += 32) {
    const float v = cand_val[m * ncand + i];
    const int id = cand_idx[m * ncand + i];
    if (v > best || (v == best && id < bi)) {
      best = v;
      bi = id;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) {
      best = ov;
      bi = oi;
    }
  }
  if (threadIdx.x == 0) {
    if (out_val) out_val[m] = best;
    out_idx[m] = bi;
  }
}

__global__ void bump_epoch_kernel(uint32_t* epoch) { *epoch += 1u; }

__global__ void add_int_kernel(int* p, int n, int delta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] += delta;
}

__global__ void copy_int_kernel(const int* src, int* dst, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[i];
}

// Input of the multi-token predictor: out[m] = [ norm_e(embed[tokens[m]]) | norm_h(hidden[m]) ], both (1 + gamma) RMSNorms.
// blockIdx.y picks the half.
__global__ void __launch_bounds__(256) mtp_concat_norm_kernel(const int* tokens, const bf16* table, const bf16* hidden, int K,
                                                              const float* gamma_e, const float* gamma_h, float eps, bf16* out) {
  extern __shared__ float row[];
  __shared__ float red[40];
  const int m = blockIdx.x, half = blockIdx.y;
  const bf16* src = half == 0 ? table + (size_t)tokens[m] * K : hidden + (size_t)m * K;
  const float* gamma = half == 0 ? gamma_e : gamma_h;
  float ss = 0.f;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float v = __bfloat162float(src[k]);
    row[k] = v;
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float r = rsqrtf(ss / (float)K + eps);
  bf16* dst = out + (size_t)m * 2 * K + (size_t)half * K;
  for (int k = threadIdx.x; k < K; k += blockDim.x) dst[k] = __float2bfloat16(row[k] * r * (1.f + gamma[k]));
}

}  // namespace

PK_API int pk_embedding(const int* tokens, int M, const void* table, int dim, int vocab_start,
                        int vocab_rows, void* out_bf16, float* out_f32, cudaStream_t stream) {
  if (M < 1) return PK_ERR_BAD_ARG;
  PK_LAUNCH(embedding_kernel, dim3(M), dim3(256), 0, stream, tokens, (const pk::bf16*)table, dim, vocab_start, vocab_rows,
                                          (pk::bf16*)out_bf16, out_f32);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_rmsnorm(const void* x, const float* parts, int nparts, int M, int K, void* hidden_out,
                      const float* gamma, int mode, float eps, void* y, const PkWait* wait,
                      cudaStream_t stream) {
  if (M < 1 || K < 1 || (x == nullptr && parts == nullptr)) return PK_ERR_BAD_ARG;
  if (hidden_out != nullptr && hidden_out == x && parts != nullptr) {
    // in place is fine here: every element is read and written by the same thread
  }
  NormParams p{};
  p.x = (const pk::bf16*)x;
  p.parts = parts;
  p.nparts = parts ? nparts : 0;
  p.M = M;
  p.K = K;
  p.hidden_out = (pk::bf16*)hidden_out;
  p.gamma = gamma;
  p.mode = mode;
  p.eps = eps;
  p.y = (pk::bf16*)y;
  if (wait) p.wait = *wait;
  const size_t smem = (size_t)K * sizeof(float);
  if (smem > 200 * 1024) return PK_ERR_UNSUPPORTED;
  // Rows of 1024 elements or more: with shorter ones most threads of a block have none. 2000 rows of 256 / 512 / 1024, us: 6.4 / 6.6 / 7.4
  // by 16 bytes, 5.4 / 6.6 / 9.3 without; one row of 1024 2.0 / 2.9.
  const bool vec = K >= 1024 && (K & 7) == 0 && (((uintptr_t)x | (uintptr_t)parts | (uintptr_t)hidden_out | (uintptr_t)gamma | (uintptr_t)y) & 15) == 0;
  if (smem > kPlainSmem) {
    // rows from 12032 elements only; the attribute is per device, so it is simply set on every such call
    if (cudaFuncSetAttribute(vec ? rmsnorm_vec_kernel : rmsnorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
  }
  if (vec) PK_LAUNCH_PDL(rmsnorm_vec_kernel, dim3(M), dim3(256), smem, stream, p);
  else PK_LAUNCH_PDL(rmsnorm_kernel, dim3(M), dim3(256), smem, stream, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// See rmsnorm_rs_ag_kernel. `y_peer[r]` is rank r's buffer of normalised rows (peer memory for r != rank); K even.
// y = rmsnorm(x) for bf16 x [M, K] (K a multiple of 8, 16-byte aligned rows); with terms = 1 or 2 (K a multiple of 128)
// the rows are also quantised for pk_gemm_fp8 exactly as pk_quant_act_fp8 would quantise y: q [terms][m_pad][K] codes,
// scale_t [K / 128][s_ld].
PK_API int pk_rmsnorm_quant(const void* x, int M, int K, const float* gamma, int mode, float eps, void* y, int terms, void* q, int m_pad,
                            float* scale_t, int s_ld, cudaStream_t stream) {
  if (M < 1 || K < 8 || (K & 7) != 0 || x == nullptr || y == nullptr || gamma == nullptr || terms < 0 || terms > 2) return PK_ERR_BAD_ARG;
  if (((uintptr_t)x & 15) != 0 || ((uintptr_t)y & 15) != 0) return PK_ERR_BAD_ARG;
  if (terms > 0 && ((K & 127) != 0 || q == nullptr || scale_t == nullptr || m_pad < M || s_ld < M || ((uintptr_t)q & 7) != 0)) return PK_ERR_BAD_ARG;
  NormQuantParams p{(const pk::bf16*)x, M, K, gamma, mode, eps, (pk::bf16*)y, terms, (uint8_t*)q, m_pad, scale_t, s_ld};
  const size_t smem = (size_t)K * sizeof(float);
  if (smem > 200 * 1024) return PK_ERR_UNSUPPORTED;
  if (smem > kPlainSmem &&
      cudaFuncSetAttribute(rmsnorm_quant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    pk_set_last_cuda_error((int)cudaGetLastError());
    return PK_ERR_CUDA;
  }
  PK_LAUNCH_PDL(rmsnorm_quant_kernel, dim3(M), dim3(256), smem, stream, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_rmsnorm_rs_ag(void* hidden, const float* parts, int world, int rank, int rows_per_rank, int M, int K, const float* gamma,
                            int mode, float eps, void* const* y_peer, const PkWait* wait_rs, const PkPush* pub_ag, const PkWait* wait_ag,
                            int sm_count, cudaStream_t stream) {
  if (world < 1 || world > PK_MAX_RANKS || rank < 0 || rank >= world || rows_per_rank < 1 || M < 1 || K < 2 || (K & 1)) return PK_ERR_BAD_ARG;
  if (wait_rs == nullptr || pub_ag == nullptr || wait_ag == nullptr || y_peer == nullptr) return PK_ERR_BAD_ARG;
  NormAgParams p{};
  p.hidden = (pk::bf16*)hidden;
  p.parts = parts;
  p.world = world;
  p.rank = rank;
  p.rpr = rows_per_rank;
  const int lo = rank * rows_per_rank;
  p.rows_mine = lo >= M ? 0 : (M - lo < rows_per_rank ? M - lo : rows_per_rank);
  p.K = K;
  p.gamma = gamma;
  p.mode = mode;
  p.eps = eps;
  for (int r = 0; r < world; ++r) p.y_peer[r] = (pk::bf16*)y_peer[r];
  p.wait_rs = *wait_rs;
  p.pub_ag = *pub_ag;
  p.wait_ag = *wait_ag;
  const size_t smem = (size_t)K * sizeof(float);
  if (smem > 200 * 1024) return PK_ERR_UNSUPPORTED;
  if (smem > kPlainSmem &&
      cudaFuncSetAttribute(rmsnorm_rs_ag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    pk_set_last_cuda_error((int)cudaGetLastError());
    return PK_ERR_CUDA;
  }
  // at least one block even without rows: every rank publishes and waits
  int blocks = p.rows_mine > 0 ? p.rows_mine : 1;
  const int cap = (sm_count > 0 ? sm_count : 148) * 4;
  if (blocks > cap) blocks = cap;
  PK_LAUNCH(rmsnorm_rs_ag_kernel, dim3(blocks), dim3(256), smem, stream, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// tokens [M] (ids inside the replicated table), hidden bf16 [M, K] -> out bf16 [M, 2K].
PK_API int pk_mtp_concat_norm(const int* tokens, int M, const void* table, const void* hidden, int K, const float* gamma_e,
                              const float* gamma_h, float eps, void* out, cudaStream_t stream) {
  if (M < 1 || K < 1 || (size_t)K * sizeof(float) > 48 * 1024) return PK_ERR_BAD_ARG;
  PK_LAUNCH(mtp_concat_norm_kernel, dim3(M, 2), dim3(256), (size_t)K * sizeof(float), stream, tokens, (const pk::bf16*)table,
            (const pk::bf16*)hidden, K, gamma_e, gamma_h, eps, (pk::bf16*)out);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_silu_mul(const void* gate_up, int M, int inter, void* out, float limit, cudaStream_t stream) {
  silu_mul_kernel<<<dim3((inter + 255) / 256, M), 256, 0, stream>>>((const pk::bf16*)gate_up, inter,
                                                                   (pk::bf16*)out, limit);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// cand_* hold M * nblocks entries. Token ids are shifted by id_offset (vocab shard start).
PK_API int pk_argmax(const float* logits, int ld, int M, int n, int id_offset, int nblocks, float* cand_val,
                     int* cand_idx, float* out_val, int* out_idx, cudaStream_t stream) {
  if (M < 1 || n < 1 || nblocks < 1) return PK_ERR_BAD_ARG;
  PK_LAUNCH(argmax_stage1, dim3(nblocks, M), dim3(256), 0, stream, logits, ld, n, id_offset, cand_val, cand_idx);
  PK_CHECK_LAUNCH();
  if (out_idx != nullptr) {
    PK_LAUNCH(argmax_stage2, dim3(M), dim3(32), 0, stream, cand_val, cand_idx, nblocks, out_val, out_idx);
    PK_CHECK_LAUNCH();
  }
  return PK_OK;
}

PK_API int pk_argmax_merge(const float* cand_val, const int* cand_idx, int M, int ncand, float* out_val,
                           int* out_idx, cudaStream_t stream) {
  PK_LAUNCH(argmax_stage2, dim3(M), dim3(32), 0, stream, cand_val, cand_idx, ncand, out_val, out_idx);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_bump_epoch(uint32_t* epoch, cudaStream_t stream) {
  PK_LAUNCH(bump_epoch_kernel, dim3(1), dim3(1), 0, stream, epoch);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_add_int(int* p, int n, int delta, cudaStream_t stream) {
  PK_LAUNCH(add_int_kernel, dim3((n + 127) / 128), dim3(128), 0, stream, p, n, delta);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

PK_API int pk_copy_int(const int* src, int* dst, int n, cudaStream_t stream) {
  PK_LAUNCH(copy_int_kernel, dim3((n + 127) / 128), dim3(128), 0, stream, src, dst, n);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// ---------------------------------------------------------------------------------------
// Random initialisation on the device (benchmarks use random-init weights of the real
// shapes; no checkpoint file is involved) and small helpers of the decode loop.
namespace {

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__device__ __forceinline__ float gauss_from(uint64_t seed, uint64_t i) {
  const uint64_t h = splitmix64(seed ^ (i * 0xD6E8FEB86659FD93ull));
  const float u1 = ((float)(uint32_t)(h >> 40) + 1.f) * (1.f / 16777217.f);
  const float u2 = (float)(uint32_t)((h >> 8) & 0xffffffu) * (1.f / 16777216.f);
  return sqrtf(-2.f * __logf(u1)) * __cosf(6.2831853f * u2);
}

// FP8 E4M3 codes of N(0, sigma) values with one scale per 128x128 block chosen so that
// 4.5 sigma maps to the largest finite code (448); blocks get slightly different scales.
__global__ void fill_fp8_gauss_kernel(uint8_t* w, float* scale, int N, int K, float sigma, uint64_t seed) {
  const size_t total = (size_t)N * K;
  const int kb = (K + 127) >> 7;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int n = (int)(i / K), k = (int)(i % K);
    const int b = (n >> 7) * kb + (k >> 7);
    const float jitter = 1.f + 0.25f * (float)(splitmix64(seed + 77u + b) & 0xff) * (1.f / 255.f);
    const float s = sigma * 4.5f / 448.f * jitter;
    if ((n & 127) == 0 && (k & 127) == 0) scale[b] = s;
    w[i] = float_to_e4m3(gauss_from(seed, i) * sigma / s);
  }
}

__global__ void fill_bf16_gauss_kernel(bf16* w, size_t n, float mean, float sigma, uint64_t seed) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    w[i] = __float2bfloat16(mean + sigma * gauss_from(seed, i));
}

__global__ void fill_f32_gauss_kernel(float* w, size_t n, float mean, float sigma, uint64_t seed) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    w[i] = mean + sigma * gauss_from(seed, i);
}

__global__ void iota_int_kernel(int* p, int n, const int* base_dev, int base_host) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = (base_dev ? *base_dev : base_host) + i;
}

__global__ void store_token_kernel(const int* token, int* out, int* counter, int cap) {
  const int c = *counter;
  if (c < cap) out[c] = *token;
  *counter = c + 1;
}

// Besides {logit, token} every rank sends its status word: a rank whose wait ran out earlier in the step tells the
// others here, so that all ranks give the step up together (slot 31 of the rank's candidate-index row).
__global__ void cand_push_kernel(const float* val, const int* idx, int M, const PkPush push,
                                 float* const* peer_val, int* const* peer_idx, const uint32_t* status, int stride) {
  const int m = threadIdx.x;
  if (m < M) {
    for (int r = 0; r < push.world; ++r) {
      peer_val[r][push.rank * stride + m] = val[m];
      peer_idx[r][push.rank * stride + m] = idx[m];
    }
  }
  if (m == 31 && status != nullptr) {
    const int st = (int)*((const volatile uint32_t*)status);
    for (int r = 0; r < push.world; ++r) peer_idx[r][push.rank * stride + 31] = st;
  }
  publish_when_grid_done(push);
}

__global__ void cand_merge_wait_kernel(const float* cand_val, const int* cand_idx, int M, int world,
                                       const PkWait wait, int* out_idx, uint32_t* status, int stride) {
  if (threadIdx.x == 0) {
    wait_all_ranks(wait);
    if (status != nullptr && *((volatile uint32_t*)status) == 0u) {
      for (int r = 0; r < world; ++r)
        if (cand_idx[r * stride + 31] != 0) atomicCAS(status, 0u, PK_COMM_PEER_FAILED);
    }
  }
  __syncthreads();
  const int m = threadIdx.x;
  if (m >= M) return;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int r = 0; r < world; ++r) {
    const float v = cand_val[r * stride + m];
    const int id = cand_idx[r * stride + m];
    if (v > best || (v == best && id < bi)) {
      best = v;
      bi = id;
    }
  }
  out_idx[m] = bi;
}

}  // namespace

PK_API int pk_fill_fp8_gauss(void* w, float* scale, int N, int K, float sigma, uint64_t seed, cudaStream_t stream) {
  fill_fp8_gauss_kernel<<<2048, 256, 0, stream>>>((uint8_t*)w, scale, N, K, sigma, seed);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
PK_API int pk_fill_bf16_gauss(void* w, size_t n, float mean, float sigma, uint64_t seed, cudaStream_t stream) {
  fill_bf16_gauss_kernel<<<1024, 256, 0, stream>>>((pk::bf16*)w, n, mean, sigma, seed);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
PK_API int pk_fill_f32_gauss(float* w, size_t n, float mean, float sigma, uint64_t seed, cudaStream_t stream) {
  fill_f32_gauss_kernel<<<256, 256, 0, stream>>>(w, n, mean, sigma, seed);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
PK_API int pk_iota_int(int* p, int n, const int* base_dev, int base_host, cudaStream_t stream) {
  iota_int_kernel<<<(n + 127) / 128, 128, 0, stream>>>(p, n, base_dev, base_host);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
PK_API int pk_store_token(const int* token, int* out, int* counter, int cap, cudaStream_t stream) {
  PK_LAUNCH(store_token_kernel, dim3(1), dim3(1), 0, stream, token, out, counter, cap);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
// Candidate rows are `stride` (>= 32) entries apart per rank; entry 31 of a rank's index row carries its status word
// (`status` may be null: nothing is sent then).
PK_API int pk_cand_push(const float* val, const int* idx, int M, const PkPush* push, float* const* peer_val,
                        int* const* peer_idx, const uint32_t* status, int stride, cudaStream_t stream) {
  if (M > 31 || stride < 32 || push == nullptr) return PK_ERR_BAD_ARG;
  cand_push_kernel<<<1, 32, 0, stream>>>(val, idx, M, *push, peer_val, peer_idx, status, stride);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
PK_API int pk_cand_merge_wait(const float* cand_val, const int* cand_idx, int M, int world, const PkWait* wait,
                              int* out_idx, uint32_t* status, int stride, cudaStream_t stream) {
  if (M > 31 || stride < 32 || wait == nullptr) return PK_ERR_BAD_ARG;
  cand_merge_wait_kernel<<<1, 32, 0, stream>>>(cand_val, cand_idx, M, world, *wait, out_idx, status, stride);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// FP8 E4M3 block-128 weights -> bf16 (w = e4m3(code) * scale[n / 128][k / 128]); 16 weights per thread.
namespace {
__global__ void __launch_bounds__(256) fp8_to_bf16_kernel(const uint8_t* __restrict__ w, const float* __restrict__ scale, int N, int K,
                                                          pk::bf16* __restrict__ out) {
  const size_t total16 = (size_t)N * K / 16;
  const int kb = (K + 127) >> 7;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total16; i += (size_t)gridDim.x * blockDim.x) {
    const size_t e = i * 16;
    const int n = (int)(e / K), k = (int)(e % K);
    const float s = scale[(size_t)(n >> 7) * kb + (k >> 7)];
    const uint4 raw = *reinterpret_cast<const uint4*>(w + e);
    const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t packed[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = pk::e4m3x2_to_float2((uint16_t)(words[j] & 0xffffu)), b = pk::e4m3x2_to_float2((uint16_t)(words[j] >> 16));
      const __nv_bfloat162 p0 = __floats2bfloat162_rn(a.x * s, a.y * s), p1 = __floats2bfloat162_rn(b.x * s, b.y * s);
      packed[2 * j] = *reinterpret_cast<const uint32_t*>(&p0);
      packed[2 * j + 1] = *reinterpret_cast<const uint32_t*>(&p1);
    }
    uint4* o = reinterpret_cast<uint4*>(out + e);
    o[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    o[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
  }
}
}  // namespace

// K must be a multiple of 16; w and out 16-byte aligned.
PK_API int pk_fp8_to_bf16(const void* w, const float* scale, int N, int K, void* out, cudaStream_t stream) {
  if (N < 1 || K < 16 || (K & 15) != 0) return PK_ERR_BAD_ARG;
  fp8_to_bf16_kernel<<<1184, 256, 0, stream>>>((const uint8_t*)w, scale, N, K, (pk::bf16*)out);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// pool[slots[j]] = src[j] for j < n: rows of row_bytes (a multiple of 16), one warp per 512 bytes of a row.
__global__ void __launch_bounds__(256) scatter_rows_kernel(const uint4* __restrict__ src, const int* __restrict__ slots, int n, int row_vec, uint4* __restrict__ pool) {
  const int j = blockIdx.y;
  const int v = blockIdx.x * 256 + threadIdx.x;
  if (j >= n || v >= row_vec) return;
  pool[(size_t)slots[j] * row_vec + v] = src[(size_t)j * row_vec + v];
}

PK_API int pk_scatter_rows(const void* src, const int* slots, int n, int row_bytes, void* pool, cudaStream_t stream) {
  if (src == nullptr || slots == nullptr || pool == nullptr || n < 1 || row_bytes < 16 || (row_bytes & 15) != 0) return PK_ERR_BAD_ARG;
  if (((uintptr_t)src & 15) != 0 || ((uintptr_t)pool & 15) != 0 || n > 65535) return PK_ERR_BAD_ARG;
  const int row_vec = row_bytes / 16;
  scatter_rows_kernel<<<dim3((row_vec + 255) / 256, n), 256, 0, stream>>>((const uint4*)src, slots, n, row_vec, (uint4*)pool);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
