// bf16 linear layers of one to eight rows (decode): the weights are streamed once, y[M, N] = x[M, K] W[N, K]^T with fp32
// accumulation, fp32 / bf16 output or a SiLU(gate) * up epilogue. A warp owns two weight rows (a gate and its up row for
// SwiGLU) and, when there are too few rows to fill the machine, a slice of K; the slices of a block are added in a fixed
// order. The first weights are requested before the wait for the previous kernel. Weight rows from `split` on may have an input of
// their own: two products whose inputs come from the same step in one launch.
#include "../common/pk_common.cuh"

namespace {

using namespace pk;

enum { OUT_BF16 = 0, OUT_SWIGLU = 1, OUT_F32 = 2 };
constexpr int WARPS = 8;
constexpr int kMmaK = 512;       // from here on linear_rows_mma_kernel where K allows it: 1024 x 256, 1 / 8 rows 1.8 / 1.8 us, 1.4 / 2.5 without; 512 x 512 1.6 / 1.6 and 1.7 / 3.2

struct RowsParams {
  const bf16* x;
  const bf16* x2;           // input of weight rows from `split` (even) on
  int split, ldx;
  const bf16* w;
  int N, K, epi, ksplit;    // ksplit: warps of a block that share a row pair (1, 2, 4, 8)
  void* y;
  int ldy;
};

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int M, int U>
__global__ void __launch_bounds__(32 * WARPS) linear_rows_kernel(const RowsParams p) {
  __shared__ float part[WARPS][2][M];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ks = p.ksplit, per_block = WARPS / ks;
  const int groups = p.epi == OUT_SWIGLU ? p.N / 2 : (p.N + 1) / 2;
  const int g = blockIdx.x * per_block + warp / ks, sl = warp % ks;
  const bool live = g < groups;
  const int n0 = p.epi == OUT_SWIGLU ? g : 2 * g;
  const int n1 = p.epi == OUT_SWIGLU ? g + groups : min(2 * g + 1, p.N - 1);
  const bf16* w0 = p.w + (size_t)(live ? n0 : 0) * p.K;
  const bf16* w1 = p.w + (size_t)(live ? n1 : 0) * p.K;
  const bf16* x = n0 < p.split ? p.x : p.x2;
  const int stride = 256 * ks;
  int k = sl * 256 + lane * 8;
  uint4 a[U], b[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    a[u] = b[u] = make_uint4(0, 0, 0, 0);
    if (live && k + u * stride < p.K) {
      a[u] = ld_stream_u4(w0 + k + u * stride);
      b[u] = ld_stream_u4(w1 + k + u * stride);
    }
  }
  pdl_trigger();
  pdl_wait();
  float acc0[M], acc1[M];
#pragma unroll
  for (int m = 0; m < M; ++m) acc0[m] = acc1[m] = 0.f;
  while (live && k < p.K) {
    const int kn = k + U * stride;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kk = k + u * stride;
      if (kk < p.K) {
        float fa[8], fb[8];
        unpack8(a[u], fa);
        unpack8(b[u], fb);
        // refill before the arithmetic: the next stretch is in flight meanwhile
        if (kk + U * stride < p.K) {
          a[u] = ld_stream_u4(w0 + kk + U * stride);
          b[u] = ld_stream_u4(w1 + kk + U * stride);
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
          float fx[8];
          unpack8(*reinterpret_cast<const uint4*>(x + (size_t)m * p.ldx + kk), fx);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            acc0[m] = fmaf(fa[e], fx[e], acc0[m]);
            acc1[m] = fmaf(fb[e], fx[e], acc1[m]);
          }
        }
      }
    }
    k = kn;
  }
#pragma unroll
  for (int m = 0; m < M; ++m) {
    acc0[m] = warp_sum(acc0[m]);
    acc1[m] = warp_sum(acc1[m]);
  }
  if (ks > 1) {
    if (lane == 0) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        part[warp][0][m] = acc0[m];
        part[warp][1][m] = acc1[m];
      }
    }
    __syncthreads();
    if (sl == 0 && lane == 0) {
      for (int s = 1; s < ks; ++s)
#pragma unroll
        for (int m = 0; m < M; ++m) {
          acc0[m] += part[warp + s][0][m];
          acc1[m] += part[warp + s][1][m];
        }
    }
  }
  if (live && sl == 0 && lane == 0) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
      if (p.epi == OUT_SWIGLU) {
        reinterpret_cast<bf16*>(p.y)[(size_t)m * p.ldy + g] = __float2bfloat16(silu(acc0[m]) * acc1[m]);
      } else if (p.epi == OUT_F32) {
        float* y = reinterpret_cast<float*>(p.y) + (size_t)m * p.ldy;
        y[n0] = acc0[m];
        if (2 * g + 1 < p.N) y[n1] = acc1[m];
      } else {
        bf16* y = reinterpret_cast<bf16*>(p.y) + (size_t)m * p.ldy;
        y[n0] = __float2bfloat16(acc0[m]);
        if (2 * g + 1 < p.N) y[n1] = __float2bfloat16(acc1[m]);
      }
    }
  }
}

// Rows of whole steps of 64: with a multiply-add per weight and row the kernel above is bound by its instructions and by loads that
// registers hold (10304 x 4096: 1 row 27 us, 8 rows 58 us). Here a warp owns 16 weight rows as the M side of m16n8k16 products with
// the token rows as the N side: 20 and 23 us; 32000 x 4096 59 and 135 us before, 42 and 46 us (6.2 and 5.7 TB/s) now. A lane takes two
// times eight neighbouring values of a row for four products (four lanes a whole stretch of 64 bytes): which of the 64 values of
// a step a product takes is the same for both operands, so no value changes lanes. The weights come through a ring of kRing steps
// in shared memory that every lane fills for itself (`cp.async`, no barrier): prefetched into registers they were waited for together
// with the activations, 2.5 TB/s. The tensor cores cut their sums off, so every 16 products have a sum of their own and these are
// added with rounding: the error of fp32 results against 64 bits is 9e-8 at K = 4096 and 1.2e-7 at 14336 (8e-8 and 1e-7 with a
// multiply-add per weight; one running sum has 5e-7 and 1.8e-6), at the same time. Nothing is shared
// between warps but the sums of a K range that was cut, added in their order.
constexpr int kRing = 6, kDeepRing = 12;      // steps; two blocks on an SM, or one where no more are launched
constexpr size_t mma_smem(int ring) { return (size_t)WARPS * ring * 4 * 32 * 16; }

template <int RING>
__global__ void __launch_bounds__(32 * WARPS, RING == kRing ? 2 : 1) linear_rows_mma_kernel(const RowsParams p, int M) {
  extern __shared__ __align__(16) uint4 ring_smem[];
  __shared__ float part[WARPS][16][9];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ks = p.ksplit, per_block = WARPS / ks;
  const bool glu = p.epi == OUT_SWIGLU;
  const int half = p.N >> 1, span = glu ? 8 : 16, outs = glu ? half : p.N;      // outputs of a warp, of all
  const int n0 = (blockIdx.x * per_block + warp / ks) * span, sl = warp % ks;
  const bool live = n0 < outs;
  const int r0 = min(n0 + g, outs - 1), r1 = glu ? r0 + half : min(n0 + 8 + g, outs - 1);
  const bf16* wa = p.w + (size_t)r0 * p.K + t * 8;
  const bf16* wb = p.w + (size_t)r1 * p.K + t * 8;
  const bf16* x = (n0 < p.split ? p.x : p.x2) + (size_t)min(g, M - 1) * p.ldx + t * 8;
  const int steps = live ? (p.K / 64 - sl + ks - 1) / ks : 0, stride = 64 * ks;
  uint4* ring = ring_smem + warp * RING * 128 + lane;
  auto copy = [&](int s) {
    if (s < steps) {
      const int k = sl * 64 + s * stride;
      const bf16* src[4] = {wa + k, wa + k + 32, wb + k, wb + k + 32};
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + (s % RING) * 128);
#pragma unroll
      for (int i = 0; i < 4; ++i) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 512), "l"(src[i]) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < RING - 1; ++s) copy(s);
  pdl_trigger();
  pdl_wait();
  float c[4] = {}, before[4][4] = {};      // sums of the step before: they are added while this one's are under way
#pragma unroll 2
  for (int s = 0; s < steps; ++s) {
    const int k = sl * 64 + s * stride;
    const uint4 x0 = *reinterpret_cast<const uint4*>(x + k), x1 = *reinterpret_cast<const uint4*>(x + k + 32);
    copy(s + RING - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
    const uint4* q = ring + (s % RING) * 128;
    const uint4 a0 = q[0], a1 = q[32], b0 = q[64], b1 = q[96];
    float d[4][4] = {};
    mma16816(d[0], a0.x, b0.x, a0.y, b0.y, x0.x, x0.y);
    mma16816(d[1], a0.z, b0.z, a0.w, b0.w, x0.z, x0.w);
    mma16816(d[2], a1.x, b1.x, a1.y, b1.y, x1.x, x1.y);
    mma16816(d[3], a1.z, b1.z, a1.w, b1.w, x1.z, x1.w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      c[i] += (before[0][i] + before[1][i]) + (before[2][i] + before[3][i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) before[j][i] = d[j][i];
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += (before[0][i] + before[1][i]) + (before[2][i] + before[3][i]);
  asm volatile("cp.async.wait_all;" ::: "memory");
  part[warp][g][2 * t] = c[0];
  part[warp][g][2 * t + 1] = c[1];
  part[warp][g + 8][2 * t] = c[2];
  part[warp][g + 8][2 * t + 1] = c[3];
  __syncthreads();
  // [group of the block][token][output]: neighbouring threads have neighbouring outputs
  for (int o = threadIdx.x; o < per_block * 8 * span; o += 32 * WARPS) {
    const int q = o / (8 * span), m = o / span % 8, r = o % span, n = (blockIdx.x * per_block + q) * span + r;
    if (m >= M || n >= outs) continue;
    float v = 0.f, u = 0.f;
    for (int w = q * ks; w < (q + 1) * ks; ++w) {
      v += part[w][r][m];
      if (glu) u += part[w][r + 8][m];
    }
    if (glu) reinterpret_cast<bf16*>(p.y)[(size_t)m * p.ldy + n] = __float2bfloat16(silu(v) * u);
    else if (p.epi == OUT_F32) reinterpret_cast<float*>(p.y)[(size_t)m * p.ldy + n] = v;
    else reinterpret_cast<bf16*>(p.y)[(size_t)m * p.ldy + n] = __float2bfloat16(v);
  }
}

}  // namespace

// As pk_linear_rows; x2 has the same stride and is the input of the weight rows from `split` (a multiple of 2) on.
PK_API int pk_linear_rows2(const void* x, const void* x2, int split, int ldx, const void* w, int M, int N, int K, int epi, void* y, int ldy, int sm_count,
                           cudaStream_t stream) {
  if (x2 == nullptr || ((uintptr_t)x2 & 15) != 0 || split < 0 || (split & 1) != 0 || (epi == OUT_SWIGLU && split < N)) return PK_ERR_BAD_ARG;
  if (M < 1 || M > 8 || N < 1 || K < 8 || (K & 7) != 0 || (ldx & 7) != 0 || ldx < K || epi < 0 || epi > 2) return PK_ERR_BAD_ARG;
  if (((uintptr_t)x & 15) != 0 || ((uintptr_t)w & 15) != 0 || (epi == OUT_SWIGLU && (N & 1) != 0)) return PK_ERR_BAD_ARG;
  if (ldy < (epi == OUT_SWIGLU ? N / 2 : N)) return PK_ERR_BAD_ARG;
  if (K >= kMmaK && (K & 63) == 0 && (split >= N || (split & 15) == 0)) {
    const int outs = epi == OUT_SWIGLU ? N / 2 : N, span = epi == OUT_SWIGLU ? 8 : 16, groups = (outs + span - 1) / span;
    int ks = 1;      // warps for two blocks on every SM, two steps of 64 in a share at least
    while (ks < WARPS && groups * ks < (sm_count > 0 ? sm_count : 148) * 2 * WARPS && K >= 128 * ks * 2) ks *= 2;
    const RowsParams p{(const pk::bf16*)x, (const pk::bf16*)x2, split, ldx, (const pk::bf16*)w, N, K, epi, ks, y, ldy};
    static PkDeviceOnce once;
    if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
      if (cudaFuncSetAttribute(linear_rows_mma_kernel<kRing>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mma_smem(kRing)) != cudaSuccess ||
          cudaFuncSetAttribute(linear_rows_mma_kernel<kDeepRing>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mma_smem(kDeepRing)) != cudaSuccess) {
        pk_set_last_cuda_error((int)cudaGetLastError());
        return PK_ERR_CUDA;
      }
      once_guard.done();
    }
    // blocks that are alone on their SM hold twice as many steps, if there are so many: 512 x 4096, one row 4.1 -> 2.8 us
    const int blocks = (groups + WARPS / ks - 1) / (WARPS / ks);
    if (blocks <= (sm_count > 0 ? sm_count : 148) && K / 64 / ks >= kRing)
      PK_LAUNCH_PDL(linear_rows_mma_kernel<kDeepRing>, dim3(blocks), dim3(32 * WARPS), mma_smem(kDeepRing), stream, p, M);
    else
      PK_LAUNCH_PDL(linear_rows_mma_kernel<kRing>, dim3(blocks), dim3(32 * WARPS), mma_smem(kRing), stream, p, M);
    return PK_OK;
  }
  const int groups = epi == OUT_SWIGLU ? N / 2 : (N + 1) / 2;
  const int want = (sm_count > 0 ? sm_count : 148) * 16;      // warps that keep enough loads in flight
  int ks = 1;
  while (ks < WARPS && groups * ks < want && K >= 512 * ks * 2) ks *= 2;
  RowsParams p{(const pk::bf16*)x, (const pk::bf16*)x2, split, ldx, (const pk::bf16*)w, N, K, epi, ks, y, ldy};
  const dim3 grid((groups + WARPS / ks - 1) / (WARPS / ks)), block(32 * WARPS);
  switch (M) {
    case 1: PK_LAUNCH_PDL((linear_rows_kernel<1, 4>), grid, block, (size_t)0, stream, p); break;
    case 2: PK_LAUNCH_PDL((linear_rows_kernel<2, 4>), grid, block, (size_t)0, stream, p); break;
    case 3: PK_LAUNCH_PDL((linear_rows_kernel<3, 2>), grid, block, (size_t)0, stream, p); break;
    case 4: PK_LAUNCH_PDL((linear_rows_kernel<4, 2>), grid, block, (size_t)0, stream, p); break;
    case 5: PK_LAUNCH_PDL((linear_rows_kernel<5, 2>), grid, block, (size_t)0, stream, p); break;
    case 6: PK_LAUNCH_PDL((linear_rows_kernel<6, 2>), grid, block, (size_t)0, stream, p); break;
    case 7: PK_LAUNCH_PDL((linear_rows_kernel<7, 2>), grid, block, (size_t)0, stream, p); break;
    default: PK_LAUNCH_PDL((linear_rows_kernel<8, 2>), grid, block, (size_t)0, stream, p); break;
  }
  return PK_OK;
}

// x [M <= 8, K] bf16 rows (stride ldx, K and ldx multiples of 8, 16-byte aligned), W [N, K] bf16. epi 0 bf16, 1 SwiGLU (N / 2
// gate rows, then N / 2 up rows; bf16 out), 2 fp32.
PK_API int pk_linear_rows(const void* x, int ldx, const void* w, int M, int N, int K, int epi, void* y, int ldy, int sm_count, cudaStream_t stream) {
  return pk_linear_rows2(x, x, (N + 1) & ~1, ldx, w, M, N, K, epi, y, ldy, sm_count, stream);
}
