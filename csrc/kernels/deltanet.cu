// Gated DeltaNet linear attention: causal depthwise conv + SiLU, gates, L2-normalised
// delta-rule state update, gated RMSNorm -- one launch per layer for 1..S tokens.
//
// Per value head h (key head hk = h / (value_heads / key_heads)) and token t:
//   c      = silu(conv4(tail, x_t))                      for the q, k and v channels
//   q, k   = c_q / sqrt(|c_q|^2 + 1e-6), c_k / sqrt(|c_k|^2 + 1e-6)
//   g      = -exp(A_log[h]) * softplus(a_t[h] + dt_bias[h]),   beta = sigmoid(b_t[h])
//   S     <- S * exp(g);  delta = (v - S^T k) * beta;  S <- S + k (x) delta
//   o      = S^T q / sqrt(key_head_dim)
//   out    = o * rsqrt(mean(o^2) + eps) * gamma * silu(z_t)
// which is the recurrence of the reference engine (cpp_engine/cuda/qwen_half_ops.cu:746-930,
// 711-730). There the steps are six kernels and the prefill form keeps a 128-float state
// column per thread; here the state lives in registers for the whole token run, and the
// projections arrive packed from one GEMM.
#include <cooperative_groups.h>

#include "../common/pk_common.cuh"

namespace {

using namespace pk;

constexpr int kDk = 128;  // key head dim
constexpr int kDv = 128;  // value head dim
constexpr int kThreads = 128;
constexpr int kCols = 32;      // of a value head's state: a block's
constexpr int kBatch = 16;     // tokens between two exchanges
constexpr int kConv = 4;

struct DeltaParams {
  const bf16* proj;    // [T, ld]: q(KD) | k(KD) | v(VD) | z(VD) | a(Hv) | b(Hv)
  int ld;
  int T;
  int key_heads, value_heads;  // local (per rank) head counts
  const float* conv_w;  // [2*KD + VD, 4], tap 3 multiplies the newest input
  float* conv_state;    // [2*KD + VD, 3], oldest first
  const float* A_log;   // [Hv]
  const float* dt_bias; // [Hv]
  const float* norm_w;  // [Dv]
  float eps;
  float* state;         // [Hv, Dk, Dv]
  bf16* out;            // [T, VD]
};

// The columns of a state do not depend on one another but for the norm of the output: a block has 32 columns of a value head, and
// the blocks of a key head (four per value head) are a cluster. What all tokens need but no state (conv, norms of q and k, gates) is
// computed for a batch of tokens at once; the recurrence itself then has no barrier: a thread has 32 rows of one column, four
// neighbouring lanes the whole column. Sums of squares of the outputs go between the blocks once per batch.
// A step of one token does the same arithmetic as that token in a longer run. Bound by the loads at the start and by the chain of a
// token's sums and updates (0.8 us a token). 16 key heads, 32 value heads, us (before: one block per key head, five barriers a token,
// every thread the whole k . q): 5 tokens 26.0 -> 10.1, 13 tokens 57.7 -> 16.6.
__global__ void __launch_bounds__(kThreads) deltanet_seq_kernel(const DeltaParams p) {
  namespace cg = cooperative_groups;
  pk::pdl_wait();
  pk::pdl_trigger();
  const cg::cluster_group cluster = cg::this_cluster();
  const int rep = p.value_heads / p.key_heads, rank = blockIdx.x % (4 * rep), hk = blockIdx.x / (4 * rep);
  const int vh = rank >> 2, c0 = (rank & 3) * kCols, h = hk * rep + vh;
  const int KD = p.key_heads * kDk, VD = p.value_heads * kDv;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rg = lane & 3, cc = warp * 8 + (lane >> 2);

  __shared__ __align__(16) float s_q[kBatch][kDk], s_k[kBatch][kDk];
  __shared__ float s_v[kBatch][kCols], s_o[kBatch][kCols];
  __shared__ float s_decay[kBatch], s_beta[kBatch], s_kq[kBatch];
  __shared__ float s_ss[2][kBatch];

  // conv channels: a thread's in q, k and (32 threads) v
  const int ch[3] = {hk * kDk + tid, KD + hk * kDk + tid, 2 * KD + h * kDv + c0 + (tid & (kCols - 1))};
  const bool has_v = tid < kCols;
  float cw[3][kConv], cs[3][kConv - 1];
#pragma unroll
  for (int u = 0; u < 3; ++u) {
#pragma unroll
    for (int j = 0; j < kConv; ++j) cw[u][j] = p.conv_w[(size_t)ch[u] * kConv + j];
#pragma unroll
    for (int j = 0; j < kConv - 1; ++j) cs[u][j] = p.conv_state[(size_t)ch[u] * (kConv - 1) + j];
  }
  // rows 16 i + 4 rg + e of the thread's column: a float4 of q or k is then one pass for the warp
  float S[32];
  float* sp = p.state + ((size_t)h * kDk + rg * 4) * kDv + c0 + cc;
#pragma unroll
  for (int i = 0; i < 32; ++i) S[i] = sp[(size_t)((i >> 2) * 16 + (i & 3)) * kDv];
  const float a_neg = -__expf(p.A_log[h]), dtb = p.dt_bias[h], gam = p.norm_w[c0 + lane], qscale = rsqrtf((float)kDk);

  for (int t0 = 0, buf = 0; t0 < p.T; t0 += kBatch, buf ^= 1) {
    const int n = min(kBatch, p.T - t0);
    const bf16* rows = p.proj + (size_t)t0 * p.ld;
    // ---- conv + SiLU, gates; a batch's loads are on their way together ----
    bf16 z[kBatch / 4];
#pragma unroll
    for (int i = 0; i < kBatch / 4; ++i)
      if (warp + 4 * i < n) z[i] = rows[(size_t)(warp + 4 * i) * p.ld + 2 * KD + VD + h * kDv + c0 + lane];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      if (u == 2 && !has_v) continue;
      bf16 x[kBatch];
#pragma unroll
      for (int t = 0; t < kBatch; ++t)
        if (t < n) x[t] = rows[(size_t)t * p.ld + ch[u]];
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        if (t >= n) break;
        const float xn = __bfloat162float(x[t]);
        float y = cw[u][0] * cs[u][0] + cw[u][1] * cs[u][1] + cw[u][2] * cs[u][2] + cw[u][3] * xn;
        cs[u][0] = cs[u][1];
        cs[u][1] = cs[u][2];
        cs[u][2] = xn;
        // Activations are 16 bit between the reference's kernels; keep that rounding.
        y = __bfloat162float(__float2bfloat16(silu(y)));
        (u == 0 ? s_q[t][tid] : u == 1 ? s_k[t][tid] : s_v[t][tid & (kCols - 1)]) = y;
      }
    }
    if (tid >= kThreads - kBatch && tid - (kThreads - kBatch) < n) {
      const int t = tid - (kThreads - kBatch);
      const bf16* row = rows + (size_t)t * p.ld + 2 * KD + 2 * VD + h;
      s_decay[t] = __expf(a_neg * softplusf_(__bfloat162float(row[0]) + dtb));
      s_beta[t] = sigmoidf_(__bfloat162float(row[p.value_heads]));
    }
    __syncthreads();
    // ---- L2 norms, k . q ----
    for (int t = warp; t < n; t += kThreads / 32) {
      float4 q = *reinterpret_cast<const float4*>(&s_q[t][4 * lane]), k = *reinterpret_cast<const float4*>(&s_k[t][4 * lane]);
      const float qn = rsqrtf(warp_sum(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w) + 1e-6f) * qscale;
      const float kn = rsqrtf(warp_sum(k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w) + 1e-6f);
      q = make_float4(q.x * qn, q.y * qn, q.z * qn, q.w * qn);
      k = make_float4(k.x * kn, k.y * kn, k.z * kn, k.w * kn);
      *reinterpret_cast<float4*>(&s_q[t][4 * lane]) = q;
      *reinterpret_cast<float4*>(&s_k[t][4 * lane]) = k;
      const float kq = warp_sum(q.x * k.x + q.y * k.y + q.z * k.z + q.w * k.w);
      if (lane == 0) s_kq[t] = kq;
    }
    __syncthreads();
    // ---- recurrence ----
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
      // S^T k and S^T q on the un-decayed state
      float kv[2] = {0.f, 0.f}, qv[2] = {0.f, 0.f}, k[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q4 = *reinterpret_cast<const float4*>(&s_q[t][16 * i + 4 * rg]), k4 = *reinterpret_cast<const float4*>(&s_k[t][16 * i + 4 * rg]);
        k[4 * i] = k4.x;
        k[4 * i + 1] = k4.y;
        k[4 * i + 2] = k4.z;
        k[4 * i + 3] = k4.w;
        kv[i & 1] = fmaf(S[4 * i], k4.x, fmaf(S[4 * i + 1], k4.y, fmaf(S[4 * i + 2], k4.z, fmaf(S[4 * i + 3], k4.w, kv[i & 1]))));
        qv[i & 1] = fmaf(S[4 * i], q4.x, fmaf(S[4 * i + 1], q4.y, fmaf(S[4 * i + 2], q4.z, fmaf(S[4 * i + 3], q4.w, qv[i & 1]))));
      }
      float kvs = kv[0] + kv[1], qvs = qv[0] + qv[1];
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        kvs += __shfl_xor_sync(0xffffffffu, kvs, o);
        qvs += __shfl_xor_sync(0xffffffffu, qvs, o);
      }
      const float decay = s_decay[t], delta = (s_v[t][cc] - decay * kvs) * s_beta[t];
      if (rg == 0) s_o[t][cc] = decay * qvs + s_kq[t] * delta;
#pragma unroll
      for (int i = 0; i < 32; ++i) S[i] = fmaf(k[i], delta, S[i] * decay);
    }
    __syncthreads();
    // ---- gated RMSNorm over the head's value dim ----
    for (int t = warp; t < n; t += kThreads / 32) {
      const float ss = warp_sum(s_o[t][lane] * s_o[t][lane]);
      if (lane == 0) s_ss[buf][t] = ss;
    }
    cluster.sync();
#pragma unroll
    for (int i = 0; i < kBatch / 4; ++i) {
      const int t = warp + 4 * i;
      if (t >= n) break;
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) ss += *cluster.map_shared_rank(&s_ss[buf][t], vh * 4 + j);
      p.out[(size_t)(t0 + t) * VD + h * kDv + c0 + lane] = __float2bfloat16(s_o[t][lane] * rsqrtf(ss / (float)kDv + p.eps) * gam * silu(__bfloat162float(z[i])));
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < 32; ++i) sp[(size_t)((i >> 2) * 16 + (i & 3)) * kDv] = S[i];
  // The tails of q and k are the whole cluster's: its blocks have read them before the first exchange.
#pragma unroll
  for (int u = 0; u < 3; ++u)
    if (u == 2 ? has_v : rank == 0)
#pragma unroll
      for (int j = 0; j < kConv - 1; ++j) p.conv_state[(size_t)ch[u] * (kConv - 1) + j] = cs[u][j];
  cluster.sync();      // the last sums have been read
}

}  // namespace

// Runs tokens 0..T-1 in order, updating `state` and `conv_state` in place.
PK_API int pk_deltanet_seq(const void* proj, int ld, int T, int key_heads, int value_heads,
                           int key_dim, int value_dim, const float* conv_w, float* conv_state,
                           const float* A_log, const float* dt_bias, const float* norm_w, float eps,
                           float* state, void* out, cudaStream_t stream) {
  if (key_dim != kDk || value_dim != kDv) return PK_ERR_UNSUPPORTED;
  if (T < 1 || key_heads < 1 || value_heads < key_heads || value_heads % key_heads != 0) return PK_ERR_BAD_ARG;
  const int rep = value_heads / key_heads;
  if (rep > 2) return PK_ERR_UNSUPPORTED;  // a cluster has eight blocks at most
  DeltaParams p{};
  p.proj = (const pk::bf16*)proj;
  p.ld = ld;
  p.T = T;
  p.key_heads = key_heads;
  p.value_heads = value_heads;
  p.conv_w = conv_w;
  p.conv_state = conv_state;
  p.A_log = A_log;
  p.dt_bias = dt_bias;
  p.norm_w = norm_w;
  p.eps = eps;
  p.state = state;
  p.out = (pk::bf16*)out;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(key_heads * rep * 4);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = rep * 4;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pk_pdl_enabled() ? 2 : 1;
  if (const cudaError_t e = cudaLaunchKernelEx(&cfg, deltanet_seq_kernel, (const DeltaParams)p); e != cudaSuccess) {
    pk_set_last_cuda_error((int)e);
    return PK_ERR_CUDA;
  }
  return PK_OK;
}
