// GQA attention for decode and speculative verify: fused per-head RMSNorm + partial RoPE
// + KV append, split-context flash decode, and the merge that also applies the output
// gate. Behavioural counterpart in the reference: cpp_engine/cuda/qwen_half_ops.cu:932-1158
// (partial_rope, append_kv, gqa_scores / softmax / gqa_values as separate passes) and
// cpp_engine/cuda/qwen_gqa_optimized.cu:253-376 (split + merge for long contexts only).
//
// Positions are read from device memory so that one captured CUDA graph serves every
// decode step; the split count is a launch constant and empty splits return at once.
#include <algorithm>

#include "../common/pk_common.cuh"

namespace {

using namespace pk;

constexpr int kD = 128;  // head dim

struct QkParams {
  const bf16* proj;   // [M, ld]: per q head [q(D) | gate(D)], then k heads, then v heads
  int ld;
  int M, Hq, Hkv;
  const int* pos;     // [M]
  const float* q_gamma;  // [D]
  const float* k_gamma;  // [D]
  float eps;
  int rotary_dim;
  float theta;
  bf16* q_out;        // [M, Hq, D]
  bf16* kcache;       // [Hkv, ctx_cap, D] bf16, or E4M3 codes (one byte per channel) when kv_fp8
  bf16* vcache;
  int ctx_cap;
  // FP8 KV cache (reference: cpp_engine/cuda/qwen_half_ops.cu:1010-1055, append_kv_fp8_kernel): every row of a head is
  // stored as E4M3 codes with one fp32 scale per 64 channels, scale = amax / 448 (1 when the group is all zero).
  int kv_fp8;
  float* kscale;      // [Hkv, ctx_cap, D / 64]
  float* vscale;
};

// A block per row, a warp per head at a time, four neighbouring channels a lane; the angles, in 64 bits, once per row. 512 rows of 40 + 8 heads
// 29 -> 10 us (a block of 128 threads per row and head, each with angles of its own). A head's partner channels are exchanged through shared memory.
constexpr int kQkWarps = 8;
__global__ void __launch_bounds__(32 * kQkWarps) qk_norm_rope_append_kernel(const QkParams p) {
  pk::pdl_wait();
  pk::pdl_trigger();
  const int m = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = 4 * lane;
  __shared__ float2 s_cs[kD / 2];
  __shared__ float4 s_y[kQkWarps][kD / 4];
  const bf16* row = p.proj + (size_t)m * p.ld;
  const int pos = p.pos[m], hr = p.rotary_dim >> 1;
  const bool in_cache = pos >= 0 && pos < p.ctx_cap;
  auto load4 = [](const bf16* x) {
    if (((uintptr_t)x & 7) == 0) return *reinterpret_cast<const uint2*>(x);
    const uint16_t* u = reinterpret_cast<const uint16_t*>(x);
    return make_uint2(u[0] | (uint32_t)u[1] << 16, u[2] | (uint32_t)u[3] << 16);
  };
  auto unpack4 = [](const uint2& u) {
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
  };
  // A head's channels, and a key head's values: the first one's are on their way while the angles are computed.
  uint2 xn = make_uint2(0u, 0u), vn = make_uint2(0u, 0u);
  auto fetch = [&](int hh) {
    if (hh >= p.Hq + p.Hkv) return;
    const bf16* at = row + (hh < p.Hq ? hh * 2 * kD : p.Hq * kD + hh * kD) + d;
    xn = load4(at);
    if (hh >= p.Hq) vn = load4(at + p.Hkv * kD);
  };
  const int first = blockIdx.y * kQkWarps + warp;
  fetch(first);
  for (int i = threadIdx.x; i < hr; i += 32 * kQkWarps) {
    const double inv_freq = pow((double)p.theta, -2.0 * (double)i / (double)p.rotary_dim);
    double sn, cs;
    sincos((double)pos * inv_freq, &sn, &cs);
    s_cs[i] = make_float2((float)cs, (float)sn);
  }
  __syncthreads();
  for (int hh = first; hh < p.Hq + p.Hkv; hh += gridDim.y * kQkWarps) {
    const bool is_q = hh < p.Hq;
    const int hk = hh - p.Hq;
    if (hh != first) fetch(hh);
    const float4 x = unpack4(xn), v4 = unpack4(vn);
    const float* gamma = (is_q ? p.q_gamma : p.k_gamma) + d;
    const float r = rsqrtf(warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w) / (float)kD + p.eps);
    float y[4] = {x.x * r * (1.f + gamma[0]), x.y * r * (1.f + gamma[1]), x.z * r * (1.f + gamma[2]), x.w * r * (1.f + gamma[3])};
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = __bfloat162float(__float2bfloat16(y[e]));
    if (hr > 0) {
      __syncwarp();
      s_y[warp][lane] = make_float4(y[0], y[1], y[2], y[3]);
      __syncwarp();
      const float* all = reinterpret_cast<const float*>(s_y[warp]);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (d + e < p.rotary_dim) {
          const bool first = d + e < hr;
          const float2 cs = s_cs[first ? d + e : d + e - hr];
          const float other = all[first ? d + e + hr : d + e - hr];
          y[e] = first ? y[e] * cs.x - other * cs.y : y[e] * cs.x + other * cs.y;
        }
    }
    auto store4 = [&](bf16* dst, const float (&v)[4]) {
      if (((uintptr_t)dst & 7) != 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16(v[e]);
        return;
      }
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    };
    if (is_q) {
      store4(p.q_out + ((size_t)m * p.Hq + hh) * kD + d, y);
      continue;
    }
    if (!in_cache && lane == 0) PK_DEBUG_RECORD(101, pos, p.ctx_cap);   // the row is not written (below)
    const float v[4] = {v4.x, v4.y, v4.z, v4.w};
    const size_t ri = (size_t)hk * p.ctx_cap + pos;
    if (p.kv_fp8) {
      // quantise the bf16-rounded key and the value per 64 channels (16 lanes)
      float ka = 0.f, va = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        y[e] = __bfloat162float(__float2bfloat16(y[e]));
        ka = fmaxf(ka, fabsf(y[e]));
        va = fmaxf(va, fabsf(v[e]));
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        ka = fmaxf(ka, __shfl_xor_sync(0xffffffffu, ka, o));
        va = fmaxf(va, __shfl_xor_sync(0xffffffffu, va, o));
      }
      const float ks = ka > 0.f ? ka / 448.f : 1.f, vs = va > 0.f ? va / 448.f : 1.f;
      if (in_cache) {
        uint8_t *kd = reinterpret_cast<uint8_t*>(p.kcache) + ri * kD + d, *vd = reinterpret_cast<uint8_t*>(p.vcache) + ri * kD + d;
        uint32_t kc = 0, vc = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          kc |= (uint32_t)float_to_e4m3(y[e] / ks) << (8 * e);
          vc |= (uint32_t)float_to_e4m3(v[e] / vs) << (8 * e);
        }
        if ((((uintptr_t)kd | (uintptr_t)vd) & 3) == 0) {
          *reinterpret_cast<uint32_t*>(kd) = kc;
          *reinterpret_cast<uint32_t*>(vd) = vc;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            kd[e] = (uint8_t)(kc >> (8 * e));
            vd[e] = (uint8_t)(vc >> (8 * e));
          }
        }
        if ((lane & 15) == 0) {
          p.kscale[ri * 2 + (lane >> 4)] = ks;
          p.vscale[ri * 2 + (lane >> 4)] = vs;
        }
      }
    } else if (in_cache) {
      store4(p.kcache + ri * kD + d, y);
      store4(p.vcache + ri * kD + d, v);
    }
  }
}

struct DecodeParams {
  const bf16* q;       // [M, Hq, D]
  const bf16* kcache;  // [Hkv, ctx_cap, D]
  const bf16* vcache;
  const int* pos;      // [M]: row m attends keys 0..pos[m]
  int M, Hq, Hkv, ctx_cap;
  float scale;
  int nsplit;
  int window;          // 0 = full; else keys in (pos-window, pos] plus the first `sink` keys
  int sink;
  float* ws;           // [M, Hq, nsplit, D + 2]
  int kv_fp8;          // caches hold E4M3 codes with one fp32 scale per 64 channels
  const float* kscale; // [Hkv, ctx_cap, 2]
  const float* vscale;
};

// Eight consecutive channels of one cached row as they lie in memory (bf16: one 16-byte load; fp8: one 8-byte load and the scale of the
// 64-channel group the lane's channels belong to), and as floats.
struct Kv8 {
  uint4 w;
  float scale;
};
__device__ __forceinline__ Kv8 load_kv8(const void* base, const float* scale, size_t row, int l16, bool fp8) {
  Kv8 r;
  if (!fp8) {
    r.w = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(base) + row * kD + l16 * 8);
    r.scale = 0.f;
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(base) + row * kD + l16 * 8);
    r.w = make_uint4(v.x, v.y, 0u, 0u);
    r.scale = scale[row * 2 + (l16 >> 3)];
  }
  return r;
}
__device__ __forceinline__ void unpack_kv8(const Kv8& r, bool fp8, float (&f)[8]) {
  const uint32_t w[4] = {r.w.x, r.w.y, r.w.z, r.w.w};
  if (!fp8) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[2 * j] = __uint_as_float(w[j] << 16);
      f[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 a = e4m3x2_to_float2((uint16_t)(w[j] & 0xffffu)), b = e4m3x2_to_float2((uint16_t)(w[j] >> 16));
      f[4 * j] = a.x * r.scale;
      f[4 * j + 1] = a.y * r.scale;
      f[4 * j + 2] = b.x * r.scale;
      f[4 * j + 3] = b.y * r.scale;
    }
  }
}

// A split has few keys per warp, and its time was that of one load after the other: the keys and values of the AHEAD next steps are on
// their way while one is worked on. One row, 48 heads of 8 key heads, 210 keys in 8 splits: 11.5 -> 7.9 us. (The same sums in the same order.)
template <int G, int AHEAD>
__global__ void __launch_bounds__(128) gqa_decode_split_kernel(const DecodeParams p) {
  pk::pdl_wait();
  pk::pdl_trigger_few();      // 8 rows of 40 heads, 20 keys in 8 splits, with the merge: 8.0 -> 6.1 us; 5 rows, 210 keys in 16 12.1 -> 9.4
  const int hk = blockIdx.x, split = blockIdx.y, m = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l16 = lane & 15, khalf = lane >> 4;
  const int len = min(p.pos[m] + 1, p.ctx_cap);
  int per = (len + p.nsplit - 1) / p.nsplit;
  per = (per + 7) & ~7;
  const int start = split * per, end = min(len, start + per);
  const int win_lo = p.window > 0 ? max(0, len - p.window) : 0;

  float qv[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p.q + ((size_t)m * p.Hq + hk * G + g) * kD + l16 * 8);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      qv[g][2 * j] = __uint_as_float(w[j] << 16) * p.scale;
      qv[g][2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u) * p.scale;
    }
  }
  float mx[G], sum[G], acc[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    mx[g] = -INFINITY;
    sum[g] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[g][j] = 0.f;
  }

  const size_t head_row0 = (size_t)hk * p.ctx_cap;
  const bool fp8 = p.kv_fp8 != 0;
  Kv8 kr[AHEAD + 1], vr[AHEAD + 1];
  auto in_range = [&](int t) { return t < end && (p.window == 0 || t >= win_lo || t < p.sink); };
  auto fetch = [&](int t, Kv8& k, Kv8& v) {
    k.w = v.w = make_uint4(0u, 0u, 0u, 0u);
    k.scale = v.scale = 0.f;
    if (in_range(t)) {
      k = load_kv8(p.kcache, p.kscale, head_row0 + t, l16, fp8);
      v = load_kv8(p.vcache, p.vscale, head_row0 + t, l16, fp8);
    }
  };
#pragma unroll
  for (int a = 0; a < AHEAD; ++a) fetch(start + warp * 2 + khalf + 8 * a, kr[a], vr[a]);
  for (int t0 = start + warp * 2; t0 < end; t0 += 8) {
    const int t = t0 + khalf;
    const bool valid = in_range(t);
    fetch(t + 8 * AHEAD, kr[AHEAD], vr[AHEAD]);
    float kf[8], vf[8];
    unpack_kv8(kr[0], fp8, kf);
    unpack_kv8(vr[0], fp8, vf);
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) {
      kr[a] = kr[a + 1];
      vr[a] = vr[a + 1];
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) s = fmaf(qv[g][j], kf[j], s);
      s += __shfl_xor_sync(0xffffffffu, s, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (valid) {
        const float nm = fmaxf(mx[g], s);
        const float c = __expf(mx[g] - nm), e = __expf(s - nm);
        sum[g] = sum[g] * c + e;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[g][j] = fmaf(e, vf[j], acc[g][j] * c);
        mx[g] = nm;
      }
    }
  }

  // merge the two key halves of each warp, then the four warps
  __shared__ float s_m[4][G], s_l[4][G], s_acc[4][G][kD];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const float om = __shfl_xor_sync(0xffffffffu, mx[g], 16);
    const float ol = __shfl_xor_sync(0xffffffffu, sum[g], 16);
    const float nm = fmaxf(mx[g], om);
    const float c0 = mx[g] == -INFINITY ? 0.f : __expf(mx[g] - nm);
    const float c1 = om == -INFINITY ? 0.f : __expf(om - nm);
    sum[g] = sum[g] * c0 + ol * c1;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float oa = __shfl_xor_sync(0xffffffffu, acc[g][j], 16);
      acc[g][j] = acc[g][j] * c0 + oa * c1;
    }
    mx[g] = nm;
    if (khalf == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) s_acc[warp][g][l16 * 8 + j] = acc[g][j];
      if (l16 == 0) {
        s_m[warp][g] = mx[g];
        s_l[warp][g] = sum[g];
      }
    }
  }
  __syncthreads();
  const int d = threadIdx.x;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float nm = fmaxf(fmaxf(s_m[0][g], s_m[1][g]), fmaxf(s_m[2][g], s_m[3][g]));
    float l = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float c = s_m[w][g] == -INFINITY ? 0.f : __expf(s_m[w][g] - nm);
      l += s_l[w][g] * c;
      a += s_acc[w][g][d] * c;
    }
    float* o = p.ws + (((size_t)m * p.Hq + hk * G + g) * p.nsplit + split) * (kD + 2);
    o[d] = a;
    if (d == 0) {
      o[kD] = nm;
      o[kD + 1] = l;
    }
  }
}

// Up to two blocks on an SM loads ahead pay (6000 keys, 256 blocks, one / four / six query heads to a key head: 1.2, 1.11, 1.05 times as fast). More blocks hide
// one another's loads, and the registers of the loads cost some of them: 512 blocks, 1000 keys in 8 splits, without / with, one to five heads .97, .95, .93, .92, .66 of
// the speed. From six heads on as many blocks are resident either way, and it pays throughout (1.04 there).
template <int G>
cudaError_t launch_split(const DecodeParams& p, dim3 grid, cudaStream_t stream) {
  const bool ahead = G >= 6 || (long long)grid.x * grid.y * grid.z <= 2 * 148;
  return ahead ? pk_launch_ex(true, gqa_decode_split_kernel<G, 2>, grid, dim3(128), 0, stream, p) : pk_launch_ex(true, gqa_decode_split_kernel<G, 0>, grid, dim3(128), 0, stream, p);
}

struct MergeParams {
  const float* ws;   // [M, Hq, nsplit, D + 2]
  int nsplit, Hq;
  const bf16* proj;  // gate source ([M, ld], gate of head h at h*2D + D), may be null
  int ld;
  bf16* out;         // [M, Hq*D]
};

// Eight splits at a time, all their loads on the way together: one after the other they were the kernel's time. One row of 48 heads in 8
// splits 11.7 -> 7.4 us.
__global__ void __launch_bounds__(kD) gqa_merge_kernel(const MergeParams p) {
  pk::pdl_wait();
  pk::pdl_trigger();
  const int m = blockIdx.x, h = blockIdx.y, d = threadIdx.x;
  const float* w = p.ws + ((size_t)m * p.Hq + h) * p.nsplit * (kD + 2);
  const float gate = p.proj != nullptr ? __bfloat162float(p.proj[(size_t)m * p.ld + h * 2 * kD + kD + d]) : 0.f;
  float mx = -INFINITY, l = 0.f, a = 0.f;
  for (int s0 = 0; s0 < p.nsplit; s0 += 8) {
    float ms[8], ls[8], as[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const bool in = s0 + s < p.nsplit;
      const float* ws = w + (size_t)(in ? s0 + s : 0) * (kD + 2);
      ms[s] = in ? ws[kD] : -INFINITY;
      ls[s] = in ? ws[kD + 1] : 0.f;
      as[s] = in ? ws[d] : 0.f;
    }
    float nm = mx;
#pragma unroll
    for (int s = 0; s < 8; ++s) nm = fmaxf(nm, ms[s]);
    const float c0 = mx == -INFINITY ? 0.f : __expf(mx - nm);
    l *= c0;
    a *= c0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const float c = ms[s] == -INFINITY ? 0.f : __expf(ms[s] - nm);
      l += ls[s] * c;
      a += as[s] * c;
    }
    mx = nm;
  }
  float o = l > 0.f ? a / l : 0.f;
  if (p.proj != nullptr) o *= sigmoidf_(gate);
  p.out[((size_t)m * p.Hq + h) * kD + d] = __float2bfloat16(o);
}

// Whole-vector variant (MiniMax-M2): the RMS statistic runs over all heads of q (or k) together with one gamma per
// element, the rotation is the half-split form on the first rope_dim dims of every head with angles from tables
// [ctx, rope_dim / 2], and k / v go to position pos[t] of caches [Hkv, ctx_cap, 128]. Inputs are the bf16 projections.
struct FullQkParams {
  const bf16* q;   // [T, Hq * D], row stride ldq
  const bf16* k;   // [T, Hkv * D], row stride ldk
  const bf16* v;   // [T, Hkv * D], row stride ldv
  int ldq, ldk, ldv;
  int Hq, Hkv;
  const int* pos;
  const float* q_gamma;
  const float* k_gamma;
  float eps;
  int rope_dim;
  const float* cos_t;
  const float* sin_t;
  bf16* q_out;     // [T, Hq, D]
  bf16* kcache;
  bf16* vcache;
  int ctx_cap;
};

__global__ void __launch_bounds__(256) full_qk_norm_rope_append_kernel(const FullQkParams p) {
  pk::pdl_wait();
  pk::pdl_trigger_few();
  __shared__ float red[40];
  const int t = blockIdx.x, is_k = blockIdx.y, tid = threadIdx.x;
  const int H = is_k ? p.Hkv : p.Hq, n = H * kD;
  const bf16* x = is_k ? p.k + (size_t)t * p.ldk : p.q + (size_t)t * p.ldq;
  const float* gamma = is_k ? p.k_gamma : p.q_gamma;
  float ss = 0.f;
  for (int i = tid; i < n; i += 256) {
    const float v = __bfloat162float(x[i]);
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / (float)n + p.eps);
  const int pos = p.pos[t], half = p.rope_dim >> 1;
  const bool in_cache = pos >= 0 && pos < p.ctx_cap;
  if (!in_cache && threadIdx.x == 0) PK_DEBUG_RECORD(101, pos, p.ctx_cap);
  for (int i = tid; i < n; i += 256) {
    const int head = i >> 7, d = i & (kD - 1);
    float y = __bfloat162float(x[i]) * rs * gamma[i];
    if (d < p.rope_dim) {
      const int j = d < half ? d : d - half, o = d < half ? i + half : i - half;
      const float yo = __bfloat162float(x[o]) * rs * gamma[o];
      const float cs = p.cos_t[(size_t)pos * half + j], sn = p.sin_t[(size_t)pos * half + j];
      y = d < half ? y * cs - yo * sn : y * cs + yo * sn;
    }
    if (!is_k) {
      p.q_out[((size_t)t * p.Hq + head) * kD + d] = __float2bfloat16(y);
    } else if (in_cache) {
      const size_t ci = ((size_t)head * p.ctx_cap + pos) * kD + d;
      p.kcache[ci] = __float2bfloat16(y);
      p.vcache[ci] = p.v[(size_t)t * p.ldv + i];
    }
  }
}

// The same for rows of whole 16-byte pieces whose rotated halves are whole pieces as well: the row is loaded once, eight elements a
// thread, and kept in shared memory, where an element finds its partner. One row of 48 heads 7.7 -> 4.1 us, 64 rows 8.3 -> 4.5; from 256
// rows on (8.6 against 9.2 us, 512 rows 9.6 against 13.3) the form above has enough blocks to hide its loads and fewer threads without an element.
constexpr int kFullQkThreads = 512, kFullQkVecRows = 128;
__global__ void __launch_bounds__(kFullQkThreads) full_qk_norm_rope_append_vec_kernel(const FullQkParams p) {
  pk::pdl_wait();
  pk::pdl_trigger_few();
  extern __shared__ __align__(16) float xs[];      // [heads * D]
  __shared__ float red[40];
  const int t = blockIdx.x, is_k = blockIdx.y, tid = threadIdx.x;
  const int H = is_k ? p.Hkv : p.Hq, n = H * kD;
  const bf16* x = is_k ? p.k + (size_t)t * p.ldk : p.q + (size_t)t * p.ldq;
  const float* gamma = is_k ? p.k_gamma : p.q_gamma;
  const int pos = p.pos[t], half = p.rope_dim >> 1;
  float ss = 0.f;
#pragma unroll 2
  for (int i = tid * 8; i < n; i += kFullQkThreads * 8) {
    const uint4 u = *reinterpret_cast<const uint4*>(x + i);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __uint_as_float(w[j] << 16);
      v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
    *reinterpret_cast<float4*>(xs + i) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(xs + i + 4) = make_float4(v[4], v[5], v[6], v[7]);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
  }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / (float)n + p.eps);
  const bool in_cache = pos >= 0 && pos < p.ctx_cap;
  if (!in_cache && threadIdx.x == 0) PK_DEBUG_RECORD(101, pos, p.ctx_cap);
  for (int i = tid * 8; i < n; i += kFullQkThreads * 8) {
    const int head = i >> 7, d = i & (kD - 1);
    float y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = xs[i + e] * rs * gamma[i + e];
    if (d < p.rope_dim) {
      const int j = d < half ? d : d - half, o = d < half ? i + half : i - half;
      const float* cs = p.cos_t + (size_t)pos * half + j;
      const float* sn = p.sin_t + (size_t)pos * half + j;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float yo = xs[o + e] * rs * gamma[o + e];
        y[e] = d < half ? y[e] * cs[e] - yo * sn[e] : y[e] * cs[e] + yo * sn[e];
      }
    }
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 pr = __floats2bfloat162_rn(y[2 * e], y[2 * e + 1]);
      w[e] = *reinterpret_cast<const uint32_t*>(&pr);
    }
    if (!is_k) {
      *reinterpret_cast<uint4*>(p.q_out + ((size_t)t * p.Hq + head) * kD + d) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if (in_cache) {
      const size_t ci = ((size_t)head * p.ctx_cap + pos) * kD + d;
      *reinterpret_cast<uint4*>(p.kcache + ci) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(p.vcache + ci) = *reinterpret_cast<const uint4*>(p.v + (size_t)t * p.ldv + i);
    }
  }
}

}  // namespace

PK_API int pk_full_qk_norm_rope_append(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv, int T, int Hq, int Hkv,
                                       int head_dim, const int* pos,
                                       const float* q_gamma, const float* k_gamma, float eps, int rope_dim, const float* cos_t,
                                       const float* sin_t, void* q_out, void* kcache, void* vcache, int ctx_cap, cudaStream_t stream) {
  if (head_dim != kD) return PK_ERR_UNSUPPORTED;
  if (T < 1 || rope_dim < 0 || rope_dim > kD || (rope_dim & 1)) return PK_ERR_BAD_ARG;
  FullQkParams p{(const pk::bf16*)q, (const pk::bf16*)k, (const pk::bf16*)v, ldq, ldk, ldv, Hq, Hkv, pos, q_gamma, k_gamma, eps, rope_dim, cos_t, sin_t,
                 (pk::bf16*)q_out, (pk::bf16*)kcache, (pk::bf16*)vcache, ctx_cap};
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)q_out | (uintptr_t)kcache | (uintptr_t)vcache;
  const size_t smem = (size_t)(Hq > Hkv ? Hq : Hkv) * kD * sizeof(float);
  if ((at & 15) == 0 && ((ldq | ldk | ldv) & 7) == 0 && (rope_dim & 15) == 0 && smem <= kPlainSmem && T <= kFullQkVecRows)
    PK_LAUNCH_PDL(full_qk_norm_rope_append_vec_kernel, dim3(T, 2), dim3(kFullQkThreads), smem, stream, p);
  else
    PK_LAUNCH_PDL_L1(full_qk_norm_rope_append_kernel, dim3(T, 2), dim3(256), 0, stream, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

namespace {
}  // namespace

// kscale / vscale non-null: FP8 KV cache (kcache / vcache hold one E4M3 code per channel, the scales one fp32 per 64
// channels: [Hkv, ctx_cap, 2]); null: bf16 caches.
PK_API int pk_qk_norm_rope_append_kv(const void* proj, int ld, int M, int Hq, int Hkv, int head_dim,
                                     const int* pos, const float* q_gamma, const float* k_gamma, float eps,
                                     int rotary_dim, float theta, void* q_out, void* kcache, void* vcache, float* kscale,
                                     float* vscale, int ctx_cap, cudaStream_t stream) {
  if (head_dim != kD) return PK_ERR_UNSUPPORTED;
  if (M < 1 || rotary_dim < 0 || rotary_dim > kD || (rotary_dim & 1) || (kscale == nullptr) != (vscale == nullptr)) return PK_ERR_BAD_ARG;
  QkParams p{(const pk::bf16*)proj, ld, M, Hq, Hkv, pos, q_gamma, k_gamma, eps, rotary_dim, theta,
             (pk::bf16*)q_out, (pk::bf16*)kcache, (pk::bf16*)vcache, ctx_cap, kscale != nullptr ? 1 : 0, kscale, vscale};
  // Few rows: a row's heads over several blocks, up to four to an SM; more blocks cost more in angles than they gain. 40 + 8 heads, us by blocks to
  // a row (1 / 2 / 3 / 6): 38 rows 6.2 / 4.2 / 3.6 / 3.0, 64 rows 6.2 / 4.2 / 3.9 / 3.6, 149 rows 6.5 / 5.7 / 4.7 / 5.9, 256 rows 7.0 / 5.8 / 7.6 / 8.5, 400 rows
  // 9.1 / 9.3 / 10.3 / 12.8.
  const int per_row = std::max(1, std::min((Hq + Hkv + kQkWarps - 1) / kQkWarps, 4 * 148 / M));
  PK_LAUNCH_PDL(qk_norm_rope_append_kernel, dim3(M, per_row), dim3(32 * kQkWarps), 0, stream, p);
  return PK_OK;
}

PK_API int pk_qk_norm_rope_append(const void* proj, int ld, int M, int Hq, int Hkv, int head_dim,
                                  const int* pos, const float* q_gamma, const float* k_gamma, float eps,
                                  int rotary_dim, float theta, void* q_out, void* kcache, void* vcache,
                                  int ctx_cap, cudaStream_t stream) {
  return pk_qk_norm_rope_append_kv(proj, ld, M, Hq, Hkv, head_dim, pos, q_gamma, k_gamma, eps, rotary_dim, theta, q_out, kcache, vcache,
                                   nullptr, nullptr, ctx_cap, stream);
}

PK_API int pk_gqa_decode_kv(const void* q, const void* kcache, const void* vcache, const float* kscale, const float* vscale,
                            const int* pos, int M, int Hq, int Hkv, int head_dim, int ctx_cap, float scale, int nsplit,
                            int window, int sink, float* ws, const void* gate_proj, int ld, void* out, cudaStream_t stream);

PK_API int pk_gqa_decode(const void* q, const void* kcache, const void* vcache, const int* pos, int M,
                         int Hq, int Hkv, int head_dim, int ctx_cap, float scale, int nsplit, int window,
                         int sink, float* ws, const void* gate_proj, int ld, void* out,
                         cudaStream_t stream) {
  return pk_gqa_decode_kv(q, kcache, vcache, nullptr, nullptr, pos, M, Hq, Hkv, head_dim, ctx_cap, scale, nsplit, window, sink, ws,
                          gate_proj, ld, out, stream);
}

// ws must hold M * Hq * nsplit * (head_dim + 2) floats. kscale / vscale non-null: FP8 KV cache (see the append).
PK_API int pk_gqa_decode_kv(const void* q, const void* kcache, const void* vcache, const float* kscale, const float* vscale,
                            const int* pos, int M, int Hq, int Hkv, int head_dim, int ctx_cap, float scale, int nsplit,
                            int window, int sink, float* ws, const void* gate_proj, int ld, void* out, cudaStream_t stream) {
  if (head_dim != kD) return PK_ERR_UNSUPPORTED;
  if (M < 1 || nsplit < 1 || Hkv < 1 || Hq < Hkv || ctx_cap < 1) return PK_ERR_BAD_ARG;   // before any division by Hkv
  if (Hq % Hkv != 0) return PK_ERR_BAD_ARG;
  if ((kscale == nullptr) != (vscale == nullptr)) return PK_ERR_BAD_ARG;
  DecodeParams p{(const pk::bf16*)q, (const pk::bf16*)kcache, (const pk::bf16*)vcache, pos, M, Hq, Hkv,
                 ctx_cap, scale, nsplit, window, sink, ws, kscale != nullptr ? 1 : 0, kscale, vscale};
  const dim3 grid(Hkv, nsplit, M);
  cudaError_t e = cudaSuccess;
  switch (Hq / Hkv) {
    case 1: e = launch_split<1>(p, grid, stream); break;
    case 2: e = launch_split<2>(p, grid, stream); break;
    case 3: e = launch_split<3>(p, grid, stream); break;
    case 4: e = launch_split<4>(p, grid, stream); break;
    case 5: e = launch_split<5>(p, grid, stream); break;
    case 6: e = launch_split<6>(p, grid, stream); break;
    case 8: e = launch_split<8>(p, grid, stream); break;
    default: return PK_ERR_UNSUPPORTED;
  }
  if (e != cudaSuccess) {
    pk_set_last_cuda_error((int)e);
    return PK_ERR_CUDA;
  }
  PK_CHECK_LAUNCH();
  MergeParams mp{ws, nsplit, Hq, (const pk::bf16*)gate_proj, ld, (pk::bf16*)out};
  PK_LAUNCH_PDL(gqa_merge_kernel, dim3(M, Hq), dim3(kD), 0, stream, mp);
  return PK_OK;
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant: the split partials live in a fixed array inside the library
// image instead of a caller-provided workspace. Contract in pk_gqa_decode_static.h.
#include <cstdio>
#include <mutex>

#include "pk_gqa_decode_static.h"

namespace {
static __device__ __align__(256) float g_gqa_static_ws[PK_GQA_STATIC_WS_FLOATS];

constexpr int kMaxStaticDevices = 64;
float* g_gqa_static_ptr[kMaxStaticDevices] = {};   // device address of the array, per device
std::mutex g_gqa_static_mu;
thread_local char g_gqa_static_msg[192] = "";
}  // namespace

PK_API const char* pk_gqa_decode_static_error(void) { return g_gqa_static_msg; }

PK_API int pk_gqa_decode_static(const void* q, const void* kcache, const void* vcache, const int* pos, int M,
                                int Hq, int Hkv, int head_dim, int ctx_cap, float scale, int nsplit,
                                int window, int sink, const void* gate_proj, int ld, void* out,
                                cudaStream_t stream) {
  g_gqa_static_msg[0] = 0;
  if (M < 1 || Hq < 1 || nsplit < 1 || head_dim < 1) {
    snprintf(g_gqa_static_msg, sizeof g_gqa_static_msg, "pk_gqa_decode_static: M, Hq, nsplit and head_dim must be positive");
    return PK_ERR_BAD_ARG;
  }
  if (Hkv < 1 || Hq < Hkv || Hq % Hkv != 0 || ctx_cap < 1) {
    snprintf(g_gqa_static_msg, sizeof g_gqa_static_msg,
             "pk_gqa_decode_static: Hkv must be positive and divide Hq, ctx_cap must be positive (Hq %d, Hkv %d, ctx_cap %d)", Hq, Hkv,
             ctx_cap);
    return PK_ERR_BAD_ARG;
  }
  const unsigned long long need = (unsigned long long)M * Hq * nsplit * (head_dim + 2);
  if (need > (unsigned long long)PK_GQA_STATIC_WS_FLOATS) {
    snprintf(g_gqa_static_msg, sizeof g_gqa_static_msg,
             "pk_gqa_decode_static: M*Hq*nsplit*(head_dim+2) = %llu floats exceeds the fixed scratch of %d floats; "
             "use pk_gqa_decode with your own workspace",
             need, (int)PK_GQA_STATIC_WS_FLOATS);
    return PK_ERR_BAD_ARG;
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    pk_set_last_cuda_error((int)e);
    return PK_ERR_CUDA;
  }
  if (dev < 0 || dev >= kMaxStaticDevices) {
    snprintf(g_gqa_static_msg, sizeof g_gqa_static_msg, "pk_gqa_decode_static: device ordinal %d is not supported", dev);
    return PK_ERR_UNSUPPORTED;
  }
  float* ws = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_gqa_static_mu);
    ws = g_gqa_static_ptr[dev];
    if (ws == nullptr) {   // first call on this device: resolve the array's device address
      e = cudaGetSymbolAddress((void**)&ws, g_gqa_static_ws);
      if (e != cudaSuccess || ws == nullptr) {
        pk_set_last_cuda_error((int)e);
        snprintf(g_gqa_static_msg, sizeof g_gqa_static_msg, "pk_gqa_decode_static: cudaGetSymbolAddress failed (%s)",
                 cudaGetErrorString(e));
        return PK_ERR_CUDA;
      }
      g_gqa_static_ptr[dev] = ws;
    }
  }
  return pk_gqa_decode(q, kcache, vcache, pos, M, Hq, Hkv, head_dim, ctx_cap, scale, nsplit, window, sink, ws,
                       gate_proj, ld, out, stream);
}
