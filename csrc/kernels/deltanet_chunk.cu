// Chunked Gated DeltaNet scan for prefill (chunk = 64 tokens).
//
// The recurrence  S_t = e^{g_t} S_{t-1} + k_t (x) delta_t,  delta_t = beta_t (v_t - (e^{g_t} S_{t-1})^T k_t)
// is serial in t; inside a chunk it is rewritten (WY / UT transform) so that only one
// state update per chunk stays serial. With G_i the running sum of g inside the chunk,
//   A_ij = beta_i e^{G_i - G_j} (k_i . k_j)  (j < i),       (I + A) Delta = beta (V - e^{G} K S_0)
//   U = (I + A)^{-1} (beta V),  W = (I + A)^{-1} (beta e^{G} K),   Delta = U - W S_0
//   O = e^{G} Q S_0 + P Delta,  P_ij = e^{G_i - G_j} (q_i . k_j)  (j <= i)
//   S_C = e^{G_C} S_0 + (e^{G_C - G} K)^T Delta
// Everything that does not touch S (conv + SiLU, norms, gates, A, U, W, P) runs in
// parallel over (head, chunk); the state pass runs over (head, quarter of the value dim).
// The reference engine has only the token-serial form for prefill
// (cpp_engine/cuda/qwen_half_ops.cu:858-930, one 128-float state column per thread).
//
// All matrix products here are fp32 multiply-adds, a thread with 4 x 4 sums, so that shared-memory reads (which set the pace of one row or
// column a thread) take less time than they do.
#include <type_traits>

#include "../common/pk_common.cuh"

namespace {

using namespace pk;

constexpr int CH = 64;   // chunk length
constexpr int D = 128;   // key and value head dim
constexpr int KS = 132;  // padded row stride of 128-wide tiles in shared memory: neighbouring rows are four banks apart

// ---------------------------------------------------------------------------------------
// prep: conv + SiLU, L2 norms, gates, for every token in parallel

struct PrepParams {
  const bf16* proj;  // [T, ld]: q(KD) | k(KD) | v(VD) | z(VD) | a(Hv) | b(Hv)
  int ld, T, Tpad, Hk, Hv;
  const float* conv_w;      // [C, 4]
  const float* conv_state;  // [C, 3] inputs at times -3, -2, -1
  const float* A_log;
  const float* dt_bias;
  float* qn;    // [Tpad, Hk, 128] l2-normalised, times 1/sqrt(128)
  float* kn;    // [Tpad, Hk, 128]
  float* v;     // [Tpad, Hv, 128]
  float* g;     // [Tpad, Hv] log decay
  float* beta;  // [Tpad, Hv]
};

// Inputs of channels ch and ch + 1 (ch even) at time t: the projection row, or the remembered tail for t < 0.
__device__ __forceinline__ float2 conv_input2(const PrepParams& p, int t, int ch) {
  if (t >= 0) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p.proj + (size_t)t * p.ld + ch));
  return make_float2(p.conv_state[(size_t)ch * 3 + (3 + t)], p.conv_state[(size_t)(ch + 1) * 3 + (3 + t)]);
}

// One block per (eight tokens, key head): 64 threads per 128-channel segment (q, k, then the head's value heads), two adjacent channels per
// thread. A token's inputs serve the conv of the three after it, the conv's weights all eight: 512 tokens 24 -> 15 us (a block per token
// read four rows and all weights for one).
constexpr int kPrepTokens = 8;
__global__ void __launch_bounds__(256) deltanet_prep_kernel(const PrepParams p) {
  pk::pdl_wait();
  pk::pdl_trigger();
  const int t0 = blockIdx.x * kPrepTokens, hk = blockIdx.y;
  const int rep = p.Hv / p.Hk;
  const int seg = threadIdx.x >> 6, th = threadIdx.x & 63, d = th * 2;  // seg 0: q, 1: k, 2+: value heads
  const int KD = p.Hk * D, VD = p.Hv * D;
  __shared__ float s_sum[kPrepTokens][2][2];
  const int h = hk * rep + (seg - 2);
  const int ch = seg == 0 ? hk * D + d : seg == 1 ? KD + hk * D + d : 2 * KD + h * D + d;
  const float4 w0 = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch * 4);
  const float4 w1 = *reinterpret_cast<const float4*>(p.conv_w + (size_t)(ch + 1) * 4);
  float2 x[kPrepTokens + 3];
#pragma unroll
  for (int i = 0; i < kPrepTokens + 3; ++i) x[i] = t0 + i - 3 < p.T ? conv_input2(p, t0 + i - 3, ch) : make_float2(0.f, 0.f);
  if (seg >= 2 && th < kPrepTokens) {
    const int t = t0 + th;
    float gg = 0.f, bb = 0.f;
    if (t < p.T) {
      const bf16* row = p.proj + (size_t)t * p.ld;
      const float a = __bfloat162float(row[2 * KD + 2 * VD + h]);
      const float b = __bfloat162float(row[2 * KD + 2 * VD + p.Hv + h]);
      gg = -__expf(p.A_log[h]) * softplusf_(a + p.dt_bias[h]);
      bb = sigmoidf_(b);
    }
    p.g[(size_t)t * p.Hv + h] = gg;
    p.beta[(size_t)t * p.Hv + h] = bb;
  }
  float2 y[kPrepTokens];
#pragma unroll
  for (int i = 0; i < kPrepTokens; ++i) {
    const float y0 = w0.x * x[i].x + w0.y * x[i + 1].x + w0.z * x[i + 2].x + w0.w * x[i + 3].x;
    const float y1 = w1.x * x[i].y + w1.y * x[i + 1].y + w1.z * x[i + 2].y + w1.w * x[i + 3].y;
    y[i] = t0 + i < p.T ? make_float2(__bfloat162float(__float2bfloat16(silu(y0))), __bfloat162float(__float2bfloat16(silu(y1)))) : make_float2(0.f, 0.f);
  }
  if (seg >= 2) {
#pragma unroll
    for (int i = 0; i < kPrepTokens; ++i) *reinterpret_cast<float2*>(p.v + ((size_t)(t0 + i) * p.Hv + h) * D + d) = y[i];
  } else {
#pragma unroll
    for (int i = 0; i < kPrepTokens; ++i) {
      const float ss = warp_sum(y[i].x * y[i].x + y[i].y * y[i].y);
      if ((th & 31) == 0) s_sum[i][seg][th >> 5] = ss;
    }
  }
  __syncthreads();
  if (seg < 2) {
    float* dst = seg == 0 ? p.qn : p.kn;
#pragma unroll
    for (int i = 0; i < kPrepTokens; ++i) {
      const float n = rsqrtf(s_sum[i][seg][0] + s_sum[i][seg][1] + 1e-6f) * (seg == 0 ? rsqrtf((float)D) : 1.f);
      *reinterpret_cast<float2*>(dst + ((size_t)(t0 + i) * p.Hk + hk) * D + d) = make_float2(y[i].x * n, y[i].y * n);
    }
  }
}

// New conv tail = inputs of the last three tokens. Runs after prep (which reads the old tail).
__global__ void deltanet_tail_kernel(const bf16* proj, int ld, int T, int channels, float* conv_state) {
  pk::pdl_wait();
  pk::pdl_trigger();
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= channels) return;
  float nv[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int t = T - 3 + j;
    nv[j] = t >= 0 ? __bfloat162float(proj[(size_t)t * ld + ch]) : conv_state[(size_t)ch * 3 + (3 + t)];
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) conv_state[(size_t)ch * 3 + j] = nv[j];
}

// ---------------------------------------------------------------------------------------
// per (chunk, value head): G, A, U, W, P. 8 chunks of 32 heads 68 -> 37 us: the products read shared memory a value a multiply-add, and
// the substitution loaded each right-hand side behind the store of the solution before it.

struct ChunkParams {
  const float* qn; const float* kn; const float* v; const float* g; const float* beta;
  int Hk, Hv, Tpad;
  float* U;   // [Hv, Tpad, 128]
  float* W;   // [Hv, Tpad, 128]
  float* P;   // [Hv, Tpad/64, 64, 64]
  float* G;   // [Hv, Tpad] running log decay inside the chunk
};

__global__ void __launch_bounds__(256, 2) deltanet_chunk_kernel(const ChunkParams p) {
  pk::pdl_wait();
  pk::pdl_trigger();
  extern __shared__ float smem[];
  float* Ks = smem;                  // [64][132]
  float* Qs = Ks + CH * KS;          // [64][132]
  float* As = Qs + CH * KS;          // [64][64]
  float* Gs = As + CH * CH;          // [64]
  float* Bs = Gs + CH;               // [64]
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int hk = h / (p.Hv / p.Hk);
  const int t0 = c * CH;

#pragma unroll 4
  for (int i = tid; i < CH * D / 4; i += 256) {
    const int r = i >> 5, d = (i & 31) * 4;
    *reinterpret_cast<float4*>(Ks + r * KS + d) = *reinterpret_cast<const float4*>(p.kn + ((size_t)(t0 + r) * p.Hk + hk) * D + d);
    *reinterpret_cast<float4*>(Qs + r * KS + d) = *reinterpret_cast<const float4*>(p.qn + ((size_t)(t0 + r) * p.Hk + hk) * D + d);
  }
  if (tid < 32) {
    // inclusive scan of g over the 64 tokens (two per lane)
    const float g0 = p.g[(size_t)(t0 + 2 * tid) * p.Hv + h], g1 = p.g[(size_t)(t0 + 2 * tid + 1) * p.Hv + h];
    float s = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, s, o);
      if (tid >= o) s += n;
    }
    Gs[2 * tid + 1] = s;
    Gs[2 * tid] = s - g1;
    Bs[2 * tid] = p.beta[(size_t)(t0 + 2 * tid) * p.Hv + h];
    Bs[2 * tid + 1] = p.beta[(size_t)(t0 + 2 * tid + 1) * p.Hv + h];
  }
  __syncthreads();
  if (tid < CH) p.G[(size_t)h * p.Tpad + t0 + tid] = Gs[tid];

  // A and P: thread owns column j and rows i = ig + 4n
  {
    const int j = tid & 63, ig = tid >> 6;
    float accA[16], accP[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) { accA[n] = 0.f; accP[n] = 0.f; }
    // columns 32 to 63 have nothing above row 32
    auto products = [&](auto first) {
      constexpr int N0 = decltype(first)::value;
#pragma unroll 2
      for (int k = 0; k < D; k += 4) {
        const float4 kj = *reinterpret_cast<const float4*>(Ks + j * KS + k);
#pragma unroll
        for (int n = N0; n < 16; ++n) {
          const int i = ig + 4 * n;
          const float4 a = *reinterpret_cast<const float4*>(Ks + i * KS + k), b = *reinterpret_cast<const float4*>(Qs + i * KS + k);
          accA[n] = fmaf(a.w, kj.w, fmaf(a.z, kj.z, fmaf(a.y, kj.y, fmaf(a.x, kj.x, accA[n]))));
          accP[n] = fmaf(b.w, kj.w, fmaf(b.z, kj.z, fmaf(b.y, kj.y, fmaf(b.x, kj.x, accP[n]))));
        }
      }
    };
    if (j < 32) products(std::integral_constant<int, 0>());
    else products(std::integral_constant<int, 8>());
    float* Pout = p.P + (((size_t)h * (p.Tpad / CH) + c) * CH) * CH;
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      const int i = ig + 4 * n;
      const float e = __expf(Gs[i] - Gs[j]);
      As[i * CH + j] = j < i ? Bs[i] * e * accA[n] : 0.f;
      Pout[i * CH + j] = j <= i ? e * accP[n] : 0.f;
    }
  }
  __syncthreads();

  // Forward substitution, one right-hand-side column per thread: columns 0..127 are
  // beta*V (-> U), columns 128..255 are beta*e^G*K (-> W).
  {
    const int col = tid & 127;
    const bool isW = tid >= 128;
    float X[CH];
    // the right-hand sides first: behind the stores of the solution the loads would wait for one another
#pragma unroll
    for (int i = 0; i < CH; ++i) X[i] = isW ? Ks[i * KS + col] : p.v[((size_t)(t0 + i) * p.Hv + h) * D + col];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      float acc = X[i] * (isW ? Bs[i] * __expf(Gs[i]) : Bs[i]);
#pragma unroll
      for (int j4 = 0; j4 < (i + 3) / 4; ++j4) {
        const float4 a = *reinterpret_cast<const float4*>(As + i * CH + j4 * 4);
        // entries at or right of the diagonal are stored as zero
        if (j4 * 4 + 0 < i) acc = fmaf(-a.x, X[j4 * 4 + 0], acc);
        if (j4 * 4 + 1 < i) acc = fmaf(-a.y, X[j4 * 4 + 1], acc);
        if (j4 * 4 + 2 < i) acc = fmaf(-a.z, X[j4 * 4 + 2], acc);
        if (j4 * 4 + 3 < i) acc = fmaf(-a.w, X[j4 * 4 + 3], acc);
      }
      X[i] = acc;
      float* dst = (isW ? p.W : p.U) + ((size_t)h * p.Tpad + t0 + i) * D + col;
      *dst = acc;
    }
  }
}

// ---------------------------------------------------------------------------------------
// state pass: serial over chunks, parallel over (value head, 32-column slice of the state)

struct StateParams {
  const float* qn; const float* kn; const float* U; const float* W; const float* P; const float* G;
  int Hk, Hv, Tpad, nchunks;
  float* state;  // [Hv, 128, 128]
  float* O;      // [Tpad, Hv, 128]
};

constexpr int SL = 32;   // state columns per block
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One block of 16 warps per SM (190 KB of shared memory). A thread has 4 x 4 sums: lane = 4 row groups x 8 column groups, a warp 16 rows of the
// slice's 32 columns, and the warps that are left share the sums' K, whose parts are added through shared memory. A step of four
// K then takes 8 reads of 16 bytes for 64 multiply-adds (a row and a column a thread took 8 for 16). q S runs with W S, on the same
// reads of S. The operands of a chunk arrive by cp.async in the buffers that the chunk before has just finished with: W and q behind
// its Delta, P and k behind its state. q and k stay unscaled in shared memory: e^{G_i} multiplies the q S sums, e^{G_C - G_j} Delta_j.
// Bound by shared-memory reads (a 16-byte read is four passes, whatever lanes share: some 7 of 9 us a chunk, the multiply-adds 3.8) and six
// barriers. 8 chunks of 32 heads: 110 -> 75 us.
constexpr int ST = 512, PS = 68;
struct StateSmem {
  float W[CH * KS], Q[CH * KS], K[CH * KS], P[CH * PS];
  float Dl[CH * SL], Dk[CH * SL];      // Delta, e^{G_C - G} Delta
  float S[D * SL];
  float R[4 * CH * SL];                // parts of sums: [4][64][32] or [2][128][32]
  float Eq[CH], Ek[CH];
};

__device__ __forceinline__ void fma4(float (&acc)[4], float a, const float4& b) {
  acc[0] = fmaf(a, b.x, acc[0]);
  acc[1] = fmaf(a, b.y, acc[1]);
  acc[2] = fmaf(a, b.z, acc[2]);
  acc[3] = fmaf(a, b.w, acc[3]);
}
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }

__global__ void __launch_bounds__(ST) deltanet_state_kernel(const StateParams p) {
  pk::pdl_wait();
  pk::pdl_trigger();
  extern __shared__ __align__(16) float smem[];
  StateSmem& m = *reinterpret_cast<StateSmem*>(smem);
  const int h = blockIdx.x, sl = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hk = h / (p.Hv / p.Hk);
  const int rg = lane >> 3, cg = (lane & 7) * 4;                       // rows 4 e + rg of a tile, columns cg ..
  const int rt = (warp & 3) * 16, kg = warp >> 2;                      // 64 x 32 sums: row tile, quarter of K
  const int st = (warp & 7) * 16, jh = warp >> 3;                      // 128 x 32 sums: row tile, half of K
  const int orow = tid >> 3, ocol = (tid & 7) * 4;                     // a thread's place when parts are added
  float* sp = p.state + (size_t)h * D * D + sl * SL;

  auto rows128 = [&](float* dst, const float* src, size_t ld) {
    for (int i = tid; i < CH * D / 4; i += ST) cp_async16(dst + (i >> 5) * KS + (i & 31) * 4, src + (i >> 5) * ld + (i & 31) * 4);
  };
  auto issue_wq = [&](int c) {
    if (c < p.nchunks) {
      rows128(m.W, p.W + ((size_t)h * p.Tpad + (size_t)c * CH) * D, D);
      rows128(m.Q, p.qn + ((size_t)c * CH * p.Hk + hk) * D, (size_t)p.Hk * D);
    }
    cp_async_commit();
  };
  auto issue_pk = [&](int c) {
    if (c < p.nchunks) {
      const float* src = p.P + (((size_t)h * p.nchunks + c) * CH) * CH;
      for (int i = tid; i < CH * CH / 4; i += ST) cp_async16(m.P + (i >> 4) * PS + (i & 15) * 4, src + i * 4);
      rows128(m.K, p.kn + ((size_t)c * CH * p.Hk + hk) * D, (size_t)p.Hk * D);
    }
    cp_async_commit();
  };

  issue_wq(0);
  issue_pk(0);
  const bool whole = ((uintptr_t)p.state & 15) == 0;      // a caller's state can begin on any float
  for (int i = tid; i < D * SL / 4; i += ST) {
    const float* s = sp + (size_t)(i >> 3) * D + (i & 7) * 4;
    *reinterpret_cast<float4*>(m.S + i * 4) = whole ? load4(s) : make_float4(s[0], s[1], s[2], s[3]);
  }
  const float* Uc = p.U + ((size_t)h * p.Tpad + orow) * D + sl * SL + ocol;
  const float* Gc = p.G + (size_t)h * p.Tpad;
  float4 u = load4(Uc);
  float g = tid < CH ? Gc[tid] : 0.f, gC = Gc[CH - 1];

  for (int c = 0; c < p.nchunks; ++c) {
    const int t0 = c * CH;
    const float eC = __expf(gC);
    if (tid < CH) {
      m.Eq[tid] = __expf(g);
      m.Ek[tid] = __expf(gC - g);
    }
    cp_async_wait<1>();   // W and q of this chunk
    __syncthreads();

    // W S and q S
    float aw[4][4] = {}, aq[4][4] = {};
#pragma unroll 2
    for (int k = kg * 32; k < kg * 32 + 32; k += 4) {
      const float4 s0 = load4(m.S + k * SL + cg), s1 = load4(m.S + (k + 1) * SL + cg), s2 = load4(m.S + (k + 2) * SL + cg), s3 = load4(m.S + (k + 3) * SL + cg);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 w = load4(m.W + (rt + 4 * e + rg) * KS + k), q = load4(m.Q + (rt + 4 * e + rg) * KS + k);
        fma4(aw[e], w.x, s0);
        fma4(aw[e], w.y, s1);
        fma4(aw[e], w.z, s2);
        fma4(aw[e], w.w, s3);
        fma4(aq[e], q.x, s0);
        fma4(aq[e], q.y, s1);
        fma4(aq[e], q.z, s2);
        fma4(aq[e], q.w, s3);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) store4(m.R + (kg * CH + rt + 4 * e + rg) * SL + cg, aw[e]);
    __syncthreads();
    issue_wq(c + 1);

    // Delta = U - W S
    {
      float4 d = u;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float4 r = load4(m.R + (n * CH + orow) * SL + ocol);
        d = make_float4(d.x - r.x, d.y - r.y, d.z - r.z, d.w - r.w);
      }
      const float ek = m.Ek[orow];
      *reinterpret_cast<float4*>(m.Dl + orow * SL + ocol) = d;
      *reinterpret_cast<float4*>(m.Dk + orow * SL + ocol) = make_float4(d.x * ek, d.y * ek, d.z * ek, d.w * ek);
    }
    if (c + 1 < p.nchunks) {
      u = load4(Uc + (size_t)(t0 + CH) * D);
      g = tid < CH ? Gc[t0 + CH + tid] : 0.f;
      gC = Gc[t0 + 2 * CH - 1];
    }
    cp_async_wait<1>();   // P and k of this chunk
    __syncthreads();

    // O = e^{G} (q S) + P Delta
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float f = m.Eq[rt + 4 * e + rg];
#pragma unroll
      for (int i = 0; i < 4; ++i) aq[e][i] *= f;
    }
#pragma unroll
    for (int j = kg * 16; j < kg * 16 + 16; j += 4) {
      const float4 d0 = load4(m.Dl + j * SL + cg), d1 = load4(m.Dl + (j + 1) * SL + cg), d2 = load4(m.Dl + (j + 2) * SL + cg), d3 = load4(m.Dl + (j + 3) * SL + cg);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 w = load4(m.P + (rt + 4 * e + rg) * PS + j);
        fma4(aq[e], w.x, d0);
        fma4(aq[e], w.y, d1);
        fma4(aq[e], w.z, d2);
        fma4(aq[e], w.w, d3);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) store4(m.R + (kg * CH + rt + 4 * e + rg) * SL + cg, aq[e]);
    // S: k^T (e^{G_C - G} Delta), rows st + 4 rg + e
    float as[4][4] = {};
#pragma unroll 4
    for (int j = jh * 32; j < jh * 32 + 32; ++j) {
      const float4 k = load4(m.K + j * KS + st + 4 * rg), d = load4(m.Dk + j * SL + cg);
      fma4(as[0], k.x, d);
      fma4(as[1], k.y, d);
      fma4(as[2], k.z, d);
      fma4(as[3], k.w, d);
    }
    __syncthreads();
    issue_pk(c + 1);
    {
      float4 o = load4(m.R + orow * SL + ocol);
#pragma unroll
      for (int n = 1; n < 4; ++n) {
        const float4 r = load4(m.R + (n * CH + orow) * SL + ocol);
        o = make_float4(o.x + r.x, o.y + r.y, o.z + r.z, o.w + r.w);
      }
      *reinterpret_cast<float4*>(p.O + ((size_t)(t0 + orow) * p.Hv + h) * D + sl * SL + ocol) = o;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; ++e) store4(m.R + (jh * D + st + 4 * rg + e) * SL + cg, as[e]);
    __syncthreads();
    for (int i = tid; i < D * SL / 4; i += ST) {
      const float4 a = load4(m.R + i * 4), b = load4(m.R + D * SL + i * 4), s = load4(m.S + i * 4);
      *reinterpret_cast<float4*>(m.S + i * 4) =
          make_float4(fmaf(eC, s.x, a.x + b.x), fmaf(eC, s.y, a.y + b.y), fmaf(eC, s.z, a.z + b.z), fmaf(eC, s.w, a.w + b.w));
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int i = tid; i < D * SL / 4; i += ST) {
    float* s = sp + (size_t)(i >> 3) * D + (i & 7) * 4;
    const float4 v = load4(m.S + i * 4);
    if (whole) {
      *reinterpret_cast<float4*>(s) = v;
    } else {
      s[0] = v.x;
      s[1] = v.y;
      s[2] = v.z;
      s[3] = v.w;
    }
  }
}

// ---------------------------------------------------------------------------------------
// gated RMSNorm of the scan output

// One warp per (token, value head), four channels per lane.
__global__ void __launch_bounds__(256) deltanet_out_kernel(const float* O, const bf16* proj, int ld, int Hk, int Hv, int T,
                                                           const float* norm_w, float eps, bf16* out) {
  pk::pdl_wait();
  pk::pdl_trigger();
  const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= T * Hv) return;
  const int t = unit / Hv, h = unit - t * Hv, d = (threadIdx.x & 31) * 4;
  const float4 o = *reinterpret_cast<const float4*>(O + ((size_t)t * Hv + h) * D + d);
  const float ss = warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w);
  const int KD = Hk * D, VD = Hv * D;
  const uint2 zr = *reinterpret_cast<const uint2*>(proj + (size_t)t * ld + 2 * KD + VD + h * D + d);
  const float z0 = __uint_as_float(zr.x << 16), z1 = __uint_as_float(zr.x & 0xffff0000u), z2 = __uint_as_float(zr.y << 16),
              z3 = __uint_as_float(zr.y & 0xffff0000u);
  const float4 w = *reinterpret_cast<const float4*>(norm_w + d);
  const float r = rsqrtf(ss / (float)D + eps);
  __nv_bfloat162 lo = __floats2bfloat162_rn(o.x * r * w.x * silu(z0), o.y * r * w.y * silu(z1));
  __nv_bfloat162 hi = __floats2bfloat162_rn(o.z * r * w.z * silu(z2), o.w * r * w.w * silu(z3));
  uint2 packed;
  packed.x = *reinterpret_cast<uint32_t*>(&lo);
  packed.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(out + (size_t)t * VD + h * D + d) = packed;
}

}  // namespace

// Workspace floats needed for T tokens (Tpad = T rounded up to 64).
PK_API size_t pk_deltanet_chunk_workspace(int T, int key_heads, int value_heads) {
  const size_t Tpad = (size_t)((T + CH - 1) / CH) * CH;
  return Tpad * key_heads * D * 2      // qn, kn
         + Tpad * value_heads * D * 4  // v, U, W, O
         + Tpad * value_heads * 3      // g, beta, G
         + (size_t)value_heads * Tpad * CH;  // P
}

// Same contract as pk_deltanet_seq (state and conv_state advance by T tokens), but the
// work is chunk-parallel. `ws` holds pk_deltanet_chunk_workspace(T, ...) floats.
PK_API int pk_deltanet_chunked(const void* proj, int ld, int T, int key_heads, int value_heads, int key_dim,
                               int value_dim, const float* conv_w, float* conv_state, const float* A_log,
                               const float* dt_bias, const float* norm_w, float eps, float* state, void* out,
                               float* ws, cudaStream_t stream) {
  if (key_dim != D || value_dim != D) return PK_ERR_UNSUPPORTED;
  if (T < 1 || key_heads < 1 || value_heads % key_heads != 0 || ((uintptr_t)ws & 15) != 0) return PK_ERR_BAD_ARG;   // cp.async of 16 bytes
  if ((ld & 3) != 0 || ((uintptr_t)proj & 7) != 0 || ((uintptr_t)out & 7) != 0 || ((uintptr_t)norm_w & 15) != 0 || ((uintptr_t)conv_w & 15) != 0)
    return PK_ERR_BAD_ARG;   // row accesses of 8 bytes, a channel's four weights at once
  const int rep = value_heads / key_heads;
  if (rep > 2) return PK_ERR_UNSUPPORTED;
  const int nchunks = (T + CH - 1) / CH, Tpad = nchunks * CH;
  float* qn = ws;
  float* kn = qn + (size_t)Tpad * key_heads * D;
  float* v = kn + (size_t)Tpad * key_heads * D;
  float* U = v + (size_t)Tpad * value_heads * D;
  float* W = U + (size_t)Tpad * value_heads * D;
  float* O = W + (size_t)Tpad * value_heads * D;
  float* g = O + (size_t)Tpad * value_heads * D;
  float* beta = g + (size_t)Tpad * value_heads;
  float* G = beta + (size_t)Tpad * value_heads;
  float* P = G + (size_t)Tpad * value_heads;

  PrepParams pp{(const pk::bf16*)proj, ld, T, Tpad, key_heads, value_heads, conv_w, conv_state, A_log, dt_bias,
                qn, kn, v, g, beta};
  PK_LAUNCH_PDL(deltanet_prep_kernel, dim3(Tpad / kPrepTokens, key_heads), dim3(64 * (2 + rep)), 0, stream, pp);
  PK_CHECK_LAUNCH();
  const int channels = (2 * key_heads + value_heads) * D;
  PK_LAUNCH_PDL(deltanet_tail_kernel, dim3((channels + 255) / 256), dim3(256), 0, stream, (const pk::bf16*)proj, ld, T, channels, conv_state);
  PK_CHECK_LAUNCH();

  static PkDeviceOnce once;
  const size_t smem_chunk = (size_t)(2 * CH * KS + CH * CH + 2 * CH) * sizeof(float);
  const size_t smem_state = sizeof(StateSmem);
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(deltanet_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_chunk) != cudaSuccess ||
        cudaFuncSetAttribute(deltanet_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_state) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  ChunkParams cp{qn, kn, v, g, beta, key_heads, value_heads, Tpad, U, W, P, G};
  PK_LAUNCH_PDL(deltanet_chunk_kernel, dim3(nchunks, value_heads), dim3(256), smem_chunk, stream, cp);
  PK_CHECK_LAUNCH();
  StateParams sp{qn, kn, U, W, P, G, key_heads, value_heads, Tpad, nchunks, state, O};
  PK_LAUNCH_PDL(deltanet_state_kernel, dim3(value_heads, D / SL), dim3(ST), smem_state, stream, sp);
  PK_CHECK_LAUNCH();
  PK_LAUNCH_PDL(deltanet_out_kernel, dim3((T * value_heads + 7) / 8), dim3(256), 0, stream, O, (const pk::bf16*)proj, ld, key_heads, value_heads, T,
                                                                     norm_w, eps, (pk::bf16*)out);
  PK_CHECK_LAUNCH();
  return PK_OK;
}
