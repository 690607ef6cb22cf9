// One to sixteen token rows with E4M3 weights (a scale per 128 x 128 block): y[M, N] = x[M, K] W[N, K]^T. A warp owns 16 weight rows as the
// M side of m16n8k16 products, the token rows are the N side; a step is the 128 weights of every row under one scale. A lane
// takes two times sixteen neighbouring codes of a row: as fp16 (exact) they are the operands of eight products, and which of the
// 128 values of a step a product takes is the same for the token rows, so no value changes lanes. Token rows are fp16 under a power
// of two per row (`pk_quant_stage_rows`): products are exact, sums fp32, the scale is applied to the sums of a step.
//
// Bound by the weights' bytes: they come through a ring of kRing steps in shared memory that every lane fills for itself
// (`cp.async`, no barrier). With the tensor memory in between (quant_umma.cu) every 128 weights of a tile pass three barriers:
// mean of the 16 products of four layers at the 27B widths, 5 rows 38 us there and 26 here, 13 rows 46 and 35 us. The first steps' weights
// are requested before the kernel waits for its predecessor, and a step's token rows behind the products of the step before: with the
// launches around them overlapped a prompt of 13 tokens went from 931 to 781 us, five verified rows from 900 to 794.
#include "../common/pk_common.cuh"

namespace {

using namespace pk;

enum { OUT_BF16 = 0, OUT_SWIGLU = 1, OUT_F32 = 2, OUT_RESID = 4 };
constexpr int WARPS = 8, kRing = 6;
constexpr size_t kSmem = (size_t)WARPS * kRing * 4 * 32 * 16;

struct RowsParams {
  const uint8_t* w;         // [N, K]
  const float* w_scale;     // [ceil(N / 128)][w_ld]
  int w_ld, N, K, M, epi, ksplit;    // ksplit: warps of a block that share 16 rows (1, 2, 4, 8)
  const __half* x;          // [M, K]
  const float* row_scale;   // [M]
  void* y;
  int ldy;
  const bf16* resid;
};

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four codes -> two words of two halves
__device__ __forceinline__ void halves(uint32_t v, uint32_t& lo, uint32_t& hi) {
  const __half2_raw a = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v & 0xffffu), __NV_E4M3);
  const __half2_raw b = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v >> 16), __NV_E4M3);
  lo = (uint32_t)a.x | (uint32_t)a.y << 16;
  hi = (uint32_t)b.x | (uint32_t)b.y << 16;
}

template <int NT>      // tiles of eight token rows
__global__ void __launch_bounds__(32 * WARPS, 2) rows_fp8_kernel(const RowsParams p) {
  extern __shared__ __align__(16) uint4 ring_smem[];
  __shared__ float part[WARPS][16][8 * NT + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ks = p.ksplit, per_block = WARPS / ks;
  const bool glu = p.epi == OUT_SWIGLU;
  const int half = p.N >> 1, span = glu ? 8 : 16, outs = glu ? half : p.N;      // outputs of a warp, of all
  const int n0 = (blockIdx.x * per_block + warp / ks) * span, sl = warp % ks;
  const bool live = n0 < outs;
  const int r0 = min(n0 + g, outs - 1), r1 = glu ? r0 + half : min(n0 + 8 + g, outs - 1);
  const uint8_t* wa = p.w + (size_t)r0 * p.K + t * 16;
  const uint8_t* wb = p.w + (size_t)r1 * p.K + t * 16;
  const float* sa = p.w_scale + (size_t)(r0 >> 7) * p.w_ld;
  const float* sb = p.w_scale + (size_t)(r1 >> 7) * p.w_ld;
  const __half* x[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) x[j] = p.x + (size_t)min(8 * j + g, p.M - 1) * p.K + t * 16;
  const int steps = live ? (p.K / 128 - sl + ks - 1) / ks : 0;
  uint4* ring = ring_smem + warp * kRing * 128 + lane;
  auto copy = [&](int s) {
    if (s < steps) {
      const int k = (sl + s * ks) * 128;
      const uint8_t* src[4] = {wa + k, wa + k + 64, wb + k, wb + k + 64};
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + (s % kRing) * 128);
#pragma unroll
      for (int i = 0; i < 4; ++i) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 512), "l"(src[i]) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kRing - 1; ++s) copy(s);
  pk::pdl_wait();      // the token rows; weights are on their way
  pk::pdl_trigger();
  float acc[NT][4] = {};
  // A step's token values are loaded behind the products of the step before that use the same registers.
  uint4 xv[2][NT][2];
  auto load_x = [&](int s, int h) {
    const int k = min(sl + s * ks, p.K / 128 - 1) * 128 + 64 * h;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      xv[h][j][0] = *reinterpret_cast<const uint4*>(x[j] + k);
      xv[h][j][1] = *reinterpret_cast<const uint4*>(x[j] + k + 8);
    }
  };
  load_x(0, 0);
  load_x(0, 1);
  float fa = __ldg(sa + min(sl, p.K / 128 - 1)), fb = __ldg(sb + min(sl, p.K / 128 - 1));
  for (int s = 0; s < steps; ++s) {
    const int kn = min(sl + (s + 1) * ks, p.K / 128 - 1);
    const float fa_next = __ldg(sa + kn), fb_next = __ldg(sb + kn);
    float c[NT][4] = {};
    copy(s + kRing - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory");
    const uint4* q = ring + (s % kRing) * 128;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 va = q[32 * h], vb = q[64 + 32 * h];
      const uint32_t a[4] = {va.x, va.y, va.z, va.w}, b[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t a0, a2, b0, b2;
        halves(a[i], a0, a2);
        halves(b[i], b0, b2);
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint4& v = xv[h][j][i >> 1];
          mma16816(c[j], a0, b0, a2, b2, (i & 1) ? v.z : v.x, (i & 1) ? v.w : v.y);
        }
      }
      load_x(s + 1, h);
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      acc[j][0] = fmaf(fa, c[j][0], acc[j][0]);
      acc[j][1] = fmaf(fa, c[j][1], acc[j][1]);
      acc[j][2] = fmaf(fb, c[j][2], acc[j][2]);
      acc[j][3] = fmaf(fb, c[j][3], acc[j][3]);
    }
    fa = fa_next;
    fb = fb_next;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    part[warp][g][8 * j + 2 * t] = acc[j][0];
    part[warp][g][8 * j + 2 * t + 1] = acc[j][1];
    part[warp][g + 8][8 * j + 2 * t] = acc[j][2];
    part[warp][g + 8][8 * j + 2 * t + 1] = acc[j][3];
  }
  __syncthreads();
  // [group of the block][token][output]: neighbouring threads have neighbouring outputs
  for (int o = threadIdx.x; o < per_block * 8 * NT * span; o += 32 * WARPS) {
    const int q = o / (8 * NT * span), m = o / span % (8 * NT), r = o % span, n = (blockIdx.x * per_block + q) * span + r;
    if (m >= p.M || n >= outs) continue;
    float v = 0.f, u = 0.f;
    for (int w = q * ks; w < (q + 1) * ks; ++w) {
      v += part[w][r][m];
      if (glu) u += part[w][r + 8][m];
    }
    const float f = p.row_scale[m];
    v *= f;
    u *= f;
    const size_t at = (size_t)m * p.ldy + n;
    if (glu) ((bf16*)p.y)[at] = __float2bfloat16(silu(v) * u);
    else if (p.epi == OUT_F32) ((float*)p.y)[at] = v;
    else if (p.epi == OUT_RESID) ((bf16*)p.y)[at] = __float2bfloat16(v + __bfloat162float(p.resid[at]));
    else ((bf16*)p.y)[at] = __float2bfloat16(v);
  }
}

}  // namespace

// `staged` [M <= 16, K] fp16 and row_scale [M] from pk_quant_stage_rows (type 20, one term); W [N, K] E4M3 codes, K a multiple of 128,
// w_scale [ceil(N / 128), w_ld]. epi 0 bf16, 1 SwiGLU bf16 (N / 2 gate rows, then as many up rows), 2 fp32, 4 bf16 with `resid` added
// (row stride ldy, may be y).
PK_API int pk_rows_fp8(const void* W, const float* w_scale, int w_ld, int M, int N, int K, const void* staged, const float* row_scale, int epi, void* y,
                       int ldy, const void* resid, int sm_count, cudaStream_t stream) {
  if (W == nullptr || w_scale == nullptr || staged == nullptr || row_scale == nullptr || y == nullptr || M < 1 || M > 16 || N < 1 || K < 128 || (K & 127) != 0 ||
      w_ld < K / 128 || ((uintptr_t)W & 15) != 0 || ((uintptr_t)staged & 15) != 0 || (epi != OUT_BF16 && epi != OUT_SWIGLU && epi != OUT_F32 && epi != OUT_RESID) ||
      (epi == OUT_SWIGLU && (N & 1) != 0) || (epi == OUT_RESID && resid == nullptr) || ldy < (epi == OUT_SWIGLU ? N / 2 : N))
    return PK_ERR_BAD_ARG;
  const int outs = epi == OUT_SWIGLU ? N / 2 : N, span = epi == OUT_SWIGLU ? 8 : 16, groups = (outs + span - 1) / span;
  int ks = 1;      // warps for two blocks on every SM, two steps in a share at least
  while (ks < WARPS && groups * ks < (sm_count > 0 ? sm_count : 148) * 2 * WARPS && K >= 256 * ks * 2) ks *= 2;
  const RowsParams p{(const uint8_t*)W, w_scale, w_ld, N, K, M, epi, ks, (const __half*)staged, row_scale, y, ldy, (const pk::bf16*)resid};
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(rows_fp8_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess ||
        cudaFuncSetAttribute(rows_fp8_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  const int blocks = (groups + WARPS / ks - 1) / (WARPS / ks);
  if (M <= 8) PK_LAUNCH_PDL(rows_fp8_kernel<1>, dim3(blocks), dim3(32 * WARPS), kSmem, stream, p);
  else PK_LAUNCH_PDL(rows_fp8_kernel<2>, dim3(blocks), dim3(32 * WARPS), kSmem, stream, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
