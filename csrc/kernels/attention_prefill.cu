// Causal GQA attention for prefill chunks on the 5th-generation tensor cores.
//
// One CTA works one (query head, tile of 128 query rows). For every 64 cached positions up to the causal limit:
//   S  = Q K^T          tcgen05.mma kind::f16, both operands K-major (head dim contiguous), fp32 S in TMEM (two buffers: S of the next
//                       step is computed while the softmax warps work on this one)
//   P  = exp2(S - m)    four softmax warps, one query row per thread: tcgen05.ld, mask, maximum, exponentials; bf16 P goes to the
//                       columns that S had, from where the next product takes it
//   O += P V            V as an MN-major operand (the cache stores a position's 128 channels contiguously, which is the MN direction
//                       of this product), O in TMEM. The reference m of a row only moves when its maximum has grown by more than a
//                       factor of 2^8; its warp then rescales O in TMEM
// K and V arrive by TMA (no multicast) into two alternating buffers each. Two CTAs are resident per SM (98 KB of shared and half of the tensor
// memory each): one's products run under the other's softmax. The output is divided by the row sum, gated (sigmoid of the projection's
// gate half) and written as bf16.
//
// Bound by the softmax (16 exponentials a cycle and SM). 1500 rows of 48 heads 155 -> 43 us, 441 rows of 40 heads behind 2560 positions 219 -> 65.
// (Before: one CTA per SM, one tile of 128 positions after the other through S, softmax with P through shared memory, P V and a fold of every
// tile's output into registers.)
//
// Every wait is bounded (status word + CTA-wide abort flag).
//
// Reference counterpart: cpp_engine/cuda/qwen_gqa_optimized.cu:106-249 (tiled prefill attention on SIMT lanes) and
// cpp_engine/cuda/qwen_half_ops.cu:1161 (gqa_prefill_f16_kernel).
#include "../common/pk_sm100.cuh"

namespace {

using namespace pk;
using namespace pk::sm100;

constexpr int kD = 128;
constexpr int kTile = 128;                 // query rows
constexpr int kKV = 64;                    // positions of a step
constexpr int kQPanel = kTile * 128;       // bytes of one 64-element-wide panel of the query tile
constexpr int kKPanel = kKV * 128;
constexpr int kThreads = 64 + 128;         // warp 0: MMA issue; warp 1: TMA; warps 2-5: softmax, epilogue
constexpr uint32_t kTmemCols = 256;        // S in two buffers of 64 columns, O
constexpr float kSlack = 8.f;              // log2 of how far a row's maximum may run ahead of its reference

struct Params {
  int M, Hq, Hkv, cap;
  const int* pos;          // [M] positions of the query rows (consecutive)
  float scale_log2;        // softmax scale * log2(e)
  const bf16* gate;        // [M, ld] or null; gate of head h at h * 256 + 128
  int ld;
  bf16* out;               // [M, Hq * 128]
  uint32_t* status;
};

struct __align__(1024) Smem {
  uint8_t q[2 * kQPanel];
  uint8_t k[2][2 * kKPanel];
  uint8_t v[2][2 * kKPanel];
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], pv_full[2];
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
};

// MN-major operand with the 128-byte swizzle: 64 contiguous elements (128 B) per row, 8 rows per 1024-byte atom; atoms
// follow each other along K every `sbo` bytes and along MN every `lbo` bytes.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3fffu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3fffu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void __launch_bounds__(kThreads, 2)
gqa_prefill_umma_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                        const Params p) {
  extern __shared__ uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, row0 = (int)(gridDim.y - 1 - blockIdx.y) * kTile;      // the last rows see most: they go first
  const int kvh = h / (p.Hq / p.Hkv);

  if (threadIdx.x == 0) {
    mbar_init(&sm.q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm.k_full[i], 1);
      mbar_init(&sm.k_empty[i], 1);
      mbar_init(&sm.v_full[i], 1);
      mbar_init(&sm.v_empty[i], 1);
      mbar_init(&sm.s_full[i], 1);
      mbar_init(&sm.p_ready[i], 4);      // one per buffer: a warp can be a step ahead of the others
      mbar_init(&sm.pv_full[i], 1);
    }
    sm.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pk::pdl_wait();
  pk::pdl_trigger();
  const uint32_t tmem_s = sm.tmem_base, tmem_o = sm.tmem_base + 2 * kKV;
  // positions are consecutive: the last row of this tile decides how far the cache is read
  const int pos0 = p.pos[0];
  const int last_row = min(row0 + kTile, p.M) - 1;
  const int n_steps = (pos0 + last_row) / kKV + 1;

  if (warp == 1) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
      mbar_arrive_expect_tx(&sm.q_full, 2 * kQPanel);
      for (int i = 0; i < 4; ++i) tma_load_2d(sm.q + i * kQPanel / 2, &tmap_q, &sm.q_full, h * kD + (i >> 1) * 64, row0 + (i & 1) * kKV);
      int k_issued = 0, v_issued = 0;
      for (int t = 0; t < n_steps; ++t) {
        const int b = t & 1, y = kvh * p.cap + t * kKV;
        if (t >= 2 && !mbar_wait(&sm.k_empty[b], ((t - 2) >> 1) & 1, &sm.abort_flag, p.status, 41)) break;
        mbar_arrive_expect_tx(&sm.k_full[b], 2 * kKPanel);
        tma_load_2d(sm.k[b], &tmap_k, &sm.k_full[b], 0, y);
        tma_load_2d(sm.k[b] + kKPanel, &tmap_k, &sm.k_full[b], 64, y);
        k_issued = t + 1;
        if (t >= 2 && !mbar_wait(&sm.v_empty[b], ((t - 2) >> 1) & 1, &sm.abort_flag, p.status, 42)) break;
        mbar_arrive_expect_tx(&sm.v_full[b], 2 * kKPanel);
        tma_load_2d(sm.v[b], &tmap_v, &sm.v_full[b], 0, y);
        tma_load_2d(sm.v[b] + kKPanel, &tmap_v, &sm.v_full[b], 64, y);
        v_issued = t + 1;
      }
      if (sm.abort_flag) {
        // gave up: let the loads in flight land before the CTA exits
        for (uint32_t i = 0; i < (1u << 20); ++i)
          if (mbar_try_wait(&sm.q_full, 0)) break;
        for (int t = max(k_issued - 2, 0); t < k_issued; ++t)
          for (uint32_t i = 0; i < (1u << 20); ++i)
            if (mbar_try_wait(&sm.k_full[t & 1], (t >> 1) & 1)) break;
        for (int t = max(v_issued - 2, 0); t < v_issued; ++t)
          for (uint32_t i = 0; i < (1u << 20); ++i)
            if (mbar_try_wait(&sm.v_full[t & 1], (t >> 1) & 1)) break;
      }
    }
    __syncwarp();
  } else if (warp == 0) {
    // ---------------- MMA issuer ----------------
    // The whole warp walks the loop and one lane issues: addresses and descriptors are then uniform, which is what the
    // instructions take.
    constexpr uint32_t idesc_s = umma_idesc(1, 1, kTile, kKV);                    // bf16 x bf16, both K-major
    constexpr uint32_t idesc_pv = umma_idesc(1, 1, kTile, kD) | (1u << 16);       // V MN-major
    const uint64_t dq = smem_desc_k_sw128(smem_u32(sm.q)), dk = smem_desc_k_sw128(smem_u32(sm.k[0])), dv = smem_desc_mn_sw128(smem_u32(sm.v[0]), kKPanel, 1024);
    const bool leader = elect_one();
    auto issue_s = [&](int t) {
      const uint32_t b = t & 1;
      if (leader) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          umma_f16(tmem_s + b * kKV, dq + ((j >> 2) * kQPanel + (j & 3) * 32 >> 4), dk + b * (2 * kKPanel >> 4) + ((j >> 2) * kKPanel + (j & 3) * 32 >> 4), idesc_s,
                   j > 0 ? 1u : 0u);
        umma_commit(&sm.s_full[b]);
        if (t + 2 < n_steps) umma_commit(&sm.k_empty[b]);
      }
      __syncwarp();
    };
    bool ok = mbar_wait_uniform(&sm.q_full, 0, &sm.abort_flag, p.status, 43) && mbar_wait_uniform(&sm.k_full[0], 0, &sm.abort_flag, p.status, 44);
    if (ok) {
      tc_fence_after();
      issue_s(0);
    }
    for (int t = 0; t < n_steps && ok; ++t) {
      const uint32_t b = t & 1;
      if (t + 1 < n_steps) {
        // the S buffer of step t + 1 is free when the product with the weights of step t - 1 is done
        if ((t > 0 && !mbar_wait_uniform(&sm.pv_full[b ^ 1], ((t - 1) >> 1) & 1, &sm.abort_flag, p.status, 45)) ||
            !mbar_wait_uniform(&sm.k_full[b ^ 1], ((t + 1) >> 1) & 1, &sm.abort_flag, p.status, 46))
          break;
        tc_fence_after();
        issue_s(t + 1);
      }
      if (!mbar_wait_uniform(&sm.v_full[b], (t >> 1) & 1, &sm.abort_flag, p.status, 47) || !mbar_wait_uniform(&sm.p_ready[b], (t >> 1) & 1, &sm.abort_flag, p.status, 48)) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_f16_ts(tmem_o, tmem_s + b * kKV + j * 8, dv + b * (2 * kKPanel >> 4) + (j * 2048 >> 4), idesc_pv, t > 0 || j > 0 ? 1u : 0u);
        umma_commit(&sm.pv_full[b]);
        if (t + 2 < n_steps) umma_commit(&sm.v_empty[b]);
      }
      __syncwarp();
    }
  } else {
    // ---------------- softmax ----------------
    const int q4 = warp & 3;                       // TMEM lane quarter of this warp
    const int r = q4 * 32 + lane;                  // query row inside the tile
    const int m = row0 + r;
    const bool row_ok = m < p.M;
    const int q_pos = pos0 + (row_ok ? m : p.M - 1);
    const uint32_t lane_off = (uint32_t)(q4 * 32) << 16, ts = tmem_s + lane_off, to = tmem_o + lane_off;
    float ref = -INFINITY, sum = 0.f;              // the row's reference (log2 units) and the sum of its weights
    bool ok = true;
    for (int t = 0; t < n_steps; ++t) {
      if (!mbar_wait_warp(&sm.s_full[t & 1], (t >> 1) & 1, &sm.abort_flag, p.status, 49)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t s[2][32];
      tmem_ld_32x32(ts + (t & 1) * kKV, s[0]);
      tmem_ld_32x32(ts + (t & 1) * kKV + 32, s[1]);
      tmem_ld_wait();
      const int c_hi = q_pos - t * kKV;            // last visible column of this row in this step
      if (__any_sync(0xffffffffu, c_hi < kKV - 1)) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > c_hi) s[c][i] = 0xff800000u;
      }
      float t4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) t4[i & 3] = fmaxf(t4[i & 3], __uint_as_float(s[c][i]));
      const float top = fmaxf(fmaxf(t4[0], t4[1]), fmaxf(t4[2], t4[3])) * p.scale_log2;
      if (ref == -INFINITY) ref = top;             // nothing was visible so far: sum and O are zero
      const bool grow = top > ref + kSlack;
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = grow ? exp2_approx(ref - top) : 1.f;
        if (t > 0) {
          if (!mbar_wait_warp(&sm.pv_full[(t - 1) & 1], ((t - 1) >> 1) & 1, &sm.abort_flag, p.status, 50)) {
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < kD / 32; ++c) {
            uint32_t x[32];
            tmem_ld_32x32(to + c * 32, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * alpha);
            tmem_st_32x32(to + c * 32, x);
          }
          tmem_st_wait();
        }
        sum *= alpha;
        if (grow) ref = top;
      }
      const float mb = ref == -INFINITY ? 0.f : ref;
      float u4[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t w[32];
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(exp2_approx(fmaf(__uint_as_float(s[c][2 * e]), p.scale_log2, -mb)),
                                                          exp2_approx(fmaf(__uint_as_float(s[c][2 * e + 1]), p.scale_log2, -mb)));
          const uint32_t b2 = *reinterpret_cast<const uint32_t*>(&pr);
          // the sum runs over the rounded values, which are what the product multiplies
          u4[e & 3] += __uint_as_float(b2 << 16) + __uint_as_float(b2 & 0xffff0000u);
          w[c * 16 + e] = b2;
        }
      sum += (u4[0] + u4[1]) + (u4[2] + u4[3]);
      tmem_st_32x32(ts + (t & 1) * kKV, w);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.p_ready[t & 1]);
    }
    // Of the products before the last only those up to the third last are known to be complete here: with a barrier for
    // even and one for odd steps that is the phase before the one waited for.
    if (ok && !mbar_wait_warp(&sm.pv_full[(n_steps - 1) & 1], ((n_steps - 1) >> 1) & 1, &sm.abort_flag, p.status, 51)) ok = false;
    tc_fence_after();
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    bf16* dst = p.out + (size_t)m * p.Hq * kD + h * kD;
    const bf16* g = p.gate ? p.gate + (size_t)m * p.ld + h * 2 * kD + kD : nullptr;
#pragma unroll 1
    for (int c = 0; c < kD / 32; ++c) {
      uint32_t x[32];
      tmem_ld_32x32(to + c * 32, x);      // all lanes of the warp take part
      tmem_ld_wait();
      if (!ok || !row_ok) continue;
      uint4 gg[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) gg[v] = g ? *reinterpret_cast<const uint4*>(g + c * 32 + v * 8) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(x[v * 8 + e]) * inv;
        if (g) {
          const uint32_t w[4] = {gg[v].x, gg[v].y, gg[v].z, gg[v].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            f[2 * e] *= 1.f / (1.f + __expf(-__uint_as_float(w[e] << 16)));
            f[2 * e + 1] *= 1.f / (1.f + __expf(-__uint_as_float(w[e] & 0xffff0000u)));
          }
        }
        uint32_t o4[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
          o4[e] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(sm.tmem_base, kTmemCols);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)sym;
  }
  return fn;
}

bool encode_rows(EncodeTiledFn encode, CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer) {
  const cuuint64_t gdim[2] = {inner, outer};
  const cuuint64_t gstride[1] = {inner * 2};
  const cuuint32_t box[2] = {64, kKV};
  const cuuint32_t estr[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// q [M, Hq, 128] bf16 (normalised and rotated), kcache / vcache [Hkv, ctx_cap, 128] bf16 already holding the rows of this
// chunk, pos [M] consecutive positions (pos[m] = pos[0] + m), full causal attention (no window). gate_proj as in
// pk_gqa_decode. Cache rows behind the last position are read (and masked): they must hold finite values.
PK_API int pk_gqa_prefill_umma(const void* q, const void* kcache, const void* vcache, const int* pos, int M, int Hq, int Hkv, int head_dim, int ctx_cap,
                               float scale, const void* gate_proj, int ld, void* out, uint32_t* status, cudaStream_t stream) {
  if (head_dim != kD) return PK_ERR_UNSUPPORTED;
  if (M < 1 || Hkv < 1 || Hq < Hkv || (Hq % Hkv) != 0 || ctx_cap < 1 || pos == nullptr || out == nullptr) return PK_ERR_BAD_ARG;
  if (((uintptr_t)q & 15) != 0 || ((uintptr_t)kcache & 15) != 0 || ((uintptr_t)vcache & 15) != 0 || ((uintptr_t)out & 15) != 0) return PK_ERR_BAD_ARG;
  if (gate_proj != nullptr && (((uintptr_t)gate_proj & 15) != 0 || (ld & 7) != 0)) return PK_ERR_BAD_ARG;
  EncodeTiledFn encode = encode_fn();
  if (encode == nullptr) return PK_ERR_UNSUPPORTED;
  CUtensorMap tq, tk, tv;
  if (!encode_rows(encode, &tq, q, (uint64_t)Hq * kD, (uint64_t)M)) return PK_ERR_CUDA;
  if (!encode_rows(encode, &tk, kcache, kD, (uint64_t)Hkv * ctx_cap)) return PK_ERR_CUDA;
  if (!encode_rows(encode, &tv, vcache, kD, (uint64_t)Hkv * ctx_cap)) return PK_ERR_CUDA;
  Params p{M, Hq, Hkv, ctx_cap, pos, scale * 1.4426950408889634f, (const pk::bf16*)gate_proj, ld, (pk::bf16*)out, status};
  const size_t smem = sizeof(Smem) + 1024;
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(gqa_prefill_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  PK_LAUNCH_PDL(gqa_prefill_umma_kernel, dim3(Hq, (M + kTile - 1) / kTile), dim3(kThreads), smem, stream, tq, tk, tv, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
