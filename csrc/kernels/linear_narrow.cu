// Products with a few dozen weight rows: y[M, N] = x[M, K] W[N, K]^T, all bf16 with fp32 sums (the gates of a DeltaNet layer: 64 rows
// of 5120). A tile GEMM has one tile for all of W and walks K alone: 35 us for 13 rows as for 512, 12 here (18 with
// eight warps of 64 rows, each lane 32 bytes in a row). The K range of 16 token
// rows and 32 weight rows is cut into sixteen warps' shares, added in their order.
//
// A lane loads two times eight consecutive values of its row for four m16n8k16 products: which of the 64 values of a step a product takes is
// the same for both operands, so no value has to change lanes. The work is a few hundred products per warp and waits for its loads:
// the tensor-memory path's set-up would cost more than the whole.
#include "../common/pk_common.cuh"

namespace {

using namespace pk;

constexpr int kWarps = 16, kTok = 16, kRows = 32;

struct NarrowParams {
  const bf16* x;
  int ldx;
  const bf16* w;
  int M, N, K;
  bf16* y;
  int ldy;
};

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(32 * kWarps) linear_narrow_kernel(const NarrowParams p) {
  __shared__ float part[kWarps][kTok][kRows + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int m0 = blockIdx.x * kTok, n0 = blockIdx.y * kRows;
  float acc[kRows / 8][4] = {};
  const bf16* xa = p.x + (size_t)min(m0 + g, p.M - 1) * p.ldx + t * 8;
  const bf16* xb = p.x + (size_t)min(m0 + g + 8, p.M - 1) * p.ldx + t * 8;
  pk::pdl_wait_for(xa, xb);
  pk::pdl_trigger();
  const bf16* wr[kRows / 8];
#pragma unroll
  for (int j = 0; j < kRows / 8; ++j) wr[j] = p.w + (size_t)min(n0 + j * 8 + g, p.N - 1) * p.K + t * 8;
#pragma unroll 2
  for (int k = warp * 64; k < p.K; k += 64 * kWarps) {
    const uint4 a0 = __ldg(reinterpret_cast<const uint4*>(xa + k)), a1 = __ldg(reinterpret_cast<const uint4*>(xa + k + 32));
    const uint4 b0 = __ldg(reinterpret_cast<const uint4*>(xb + k)), b1 = __ldg(reinterpret_cast<const uint4*>(xb + k + 32));
#pragma unroll
    for (int j = 0; j < kRows / 8; ++j) {
      const uint4 w0 = __ldg(reinterpret_cast<const uint4*>(wr[j] + k)), w1 = __ldg(reinterpret_cast<const uint4*>(wr[j] + k + 32));
      mma16816(acc[j], a0.x, b0.x, a0.y, b0.y, w0.x, w0.y);
      mma16816(acc[j], a0.z, b0.z, a0.w, b0.w, w0.z, w0.w);
      mma16816(acc[j], a1.x, b1.x, a1.y, b1.y, w1.x, w1.y);
      mma16816(acc[j], a1.z, b1.z, a1.w, b1.w, w1.z, w1.w);
    }
  }
#pragma unroll
  for (int j = 0; j < kRows / 8; ++j) {
    part[warp][g][j * 8 + 2 * t] = acc[j][0];
    part[warp][g][j * 8 + 2 * t + 1] = acc[j][1];
    part[warp][g + 8][j * 8 + 2 * t] = acc[j][2];
    part[warp][g + 8][j * 8 + 2 * t + 1] = acc[j][3];
  }
  __syncthreads();
  for (int o = threadIdx.x; o < kTok * kRows; o += 32 * kWarps) {
    const int m = o / kRows, n = o - m * kRows;
    if (m0 + m >= p.M || n0 + n >= p.N) continue;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += part[w][m][n];
    p.y[(size_t)(m0 + m) * p.ldy + n0 + n] = __float2bfloat16(s);
  }
}

}  // namespace

// x [M, K] (row stride ldx), W [N, K], y [M, N] (row stride ldy), bf16; K a multiple of 64, ldx of 8, x and W on 16 bytes.
PK_API int pk_linear_narrow(const void* x, int ldx, const void* w, int M, int N, int K, void* y, int ldy, cudaStream_t stream) {
  if (x == nullptr || w == nullptr || y == nullptr || M < 1 || N < 1 || K < 64 || (K & 63) != 0 || (ldx & 7) != 0 || ldx < K || ldy < N ||
      ((uintptr_t)x & 15) != 0 || ((uintptr_t)w & 15) != 0 || (N + kRows - 1) / kRows > 65535)
    return PK_ERR_BAD_ARG;
  const NarrowParams p{(const pk::bf16*)x, ldx, (const pk::bf16*)w, M, N, K, (pk::bf16*)y, ldy};
  PK_LAUNCH_PDL(linear_narrow_kernel, dim3((M + kTok - 1) / kTok, (N + kRows - 1) / kRows), dim3(32 * kWarps), 0, stream, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
