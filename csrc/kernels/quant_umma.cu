// Products of few token rows with quantised weights through the 5th-generation tensor cores: linear layers and routed experts on raw
// GGUF blocks, linear layers in E4M3 with a scale per 128 x 128 block.
//
// The weights are the M side of the product: a tile is 128 weight rows times up to 64 token columns (a token row takes one, or two where its
// values are two terms), so that a step with one token decodes every weight once and one with hundreds once per 64 columns; none is
// expanded in HBM. Decode warps write the INTEGER part
// of the weights (codebook entry or code times the sub-block's scale: at most 11 bits) as fp16 into the swizzled A tiles, token
// rows are fp16 under a power of two per row (`pk_quant_stage_rows`), and the fp32 factor of a block is applied when
// the block's accumulator is folded from TMEM into registers: every product of a bf16 value within 2^-24 of its row's largest is
// exact (smaller ones lose bits that fp16 has no place for) and every sum is fp32. K-quants carry a minimum per 32 weights: these
// are a second, 16-wide product per block, of the minima's codes with the sums of the token values (two fp16 terms each).
//
// Measured per layer of the MiniMax-M2 shape (256 experts of 3 x 1536 x 3072 in IQ2_XXS, top 8), experts alone: 23 tokens 1860 -> 650 us
// (kernels that decode in registers), 256 tokens 4590 -> 1215 us (decode to a bf16 scratch, bf16 GEMM), 1500 tokens 4750 -> 1470 us. Bound by
// the shared-memory pipe of the decode (77 % busy, a third of it bank conflicts of the codebook's random 8-byte reads; issue slots 67 %,
// DRAM 9 %): 0.14 ms of weights at the copy rate. One token's 8 routes: 50 + 32 -> 39 + 26 us with K in parts. E4M3, 40
// rows of 34816 x 5120: 71 us, 2.5 TB/s.
//
//   warps 0-3 (0-7 for 64 columns)  fold: TMEM -> fp32 registers with the block factors, epilogue
//   next warp                       MMA issuer
//   next warp                       token tiles by TMA (no multicast)
//   8 warps (16 for 64 columns)     decode
//
// Weights per lane stay in the order 0 2 1 3 within four (what masking two bytes of a word into two halves gives); the staged
// token rows have the same order.
#include <cuda.h>

#include "../common/pk_common.cuh"
#include "../common/pk_sm100.cuh"

namespace {

using namespace pk;
using namespace pk::sm100;

#include "gguf_codebooks.inc"

enum : int { T_IQ2_XXS = 0, T_Q4_K = 3, T_Q5_K = 4, T_E4M3 = 20 };

constexpr int BM = 128;
constexpr int kMaxGroups = 512;
constexpr uint32_t kDrainPolls = 1u << 14;      // after a wait that ran out: time for copies and products in flight, which take microseconds

template <int TYPE> struct Fmt;
// `k`: weights under one factor; `cols`: places of a staged token row for them
template <> struct Fmt<T_IQ2_XXS> { static constexpr int bytes = 66, k = 256, cols = 256; static constexpr bool mins = false; };
template <> struct Fmt<T_Q4_K> { static constexpr int bytes = 144, k = 256, cols = 320; static constexpr bool mins = true; };
template <> struct Fmt<T_Q5_K> { static constexpr int bytes = 176, k = 256, cols = 320; static constexpr bool mins = true; };
template <> struct Fmt<T_E4M3> { static constexpr int bytes = 128, k = 128, cols = 128; static constexpr bool mins = false; };

enum { OUT_BF16 = 0, OUT_SWIGLU_BF16 = 1, OUT_F32 = 2, OUT_SWIGLU_F32 = 3, OUT_RESID = 4 };

struct Params {
  const uint8_t* W;       // [n_groups * rows] raw rows
  long long rb;           // bytes of a row
  int nblk;               // blocks of a row
  int rows;               // weight rows of a group
  int n_groups;
  const int* seg;         // [n_groups + 1] first token row of every group; null: one group of M rows
  int M;
  int epi;
  float limit;            // SwiGLU clamp, 0 = off
  void* out;              // token-major
  int ldo;
  const bf16* resid;      // OUT_RESID: added, row stride ldo (may be `out`)
  const float* row_scale; // what a token row's products are multiplied by
  const float* w_scale;   // E4M3: [rows / 128][w_ld]
  int w_ld;
  int parts;              // of K, summed on their own and added in their order: by one CTA (splits 1, 16 columns) or by the last of a tile's CTAs
  int splits;             // 1 or `parts`
  float* ws;              // [tile][split][column][128]
  uint32_t* counters;     // [tile], zero between launches
  uint32_t* status;       // first wait that ran out; a launch that finds it set gives NaN
};

// IQ2_XXS with few columns has two CTAs per SM, which hide one another's waits; the others have more bytes per weight and one CTA with
// twice the decode warps and a deeper ring.
template <int TYPE, int NT>
struct Shape {
  static constexpr bool kWide = TYPE != T_IQ2_XXS || NT == 64;
  static constexpr int kFoldWarps = NT == 64 ? 8 : 4;
  static constexpr int kFoldCols = NT == 64 ? 32 : NT;
  static constexpr int kDecWarps = kWide ? 16 : 8;
  static constexpr int kRows = BM / kDecWarps;          // of a decode warp
  static constexpr int kStages = kWide ? 3 : 2;
  static constexpr int kSlots = TYPE == T_E4M3 ? 4 : 3;
  static constexpr int kABytes = 2 * BM * 128, kBBytes = 2 * NT * 128;      // a stage: 128 weights of every row, in two slabs of 64
  static constexpr int kThreads = 32 * (kFoldWarps + 2 + kDecWarps);
  static constexpr int kCtas = kWide ? 1 : 2;      // resident per SM
};

template <class S, int PITCH>
struct __align__(1024) Smem {
  uint8_t a[S::kStages][S::kABytes];
  uint8_t b[S::kStages][S::kBBytes];
  uint8_t ring[S::kSlots][BM * PITCH];
  uint64_t grid[PITCH == 68 ? 256 : 1];
  uint64_t full[S::kStages], empty[S::kStages];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t drained;
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
  uint32_t last;
  int prefix[kMaxGroups + 1];     // token tiles before each group
};

// One stretch of work: blocks [b0, b1) of a tile of 128 weight rows and up to NT columns.
struct Item {
  int group, rt, split, b0, b1, row0, cnt, tile;
};

template <int NT, int TERMS>
__device__ __forceinline__ bool item_at(const Params& p, const int* prefix, int row_tiles, int i, Item& w) {
  const int total = prefix[p.n_groups];
  w.split = i % p.splits;
  i /= p.splits;
  w.tile = i;
  w.rt = i % row_tiles;
  const int tt = i / row_tiles;
  if (tt >= total) return false;
  int lo = 0, hi = p.n_groups;      // prefix[lo] <= tt < prefix[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= tt) lo = mid;
    else hi = mid;
  }
  w.group = lo;
  const int first = p.seg ? __ldg(p.seg + lo) : 0, end = p.seg ? __ldg(p.seg + lo + 1) : p.M;
  w.row0 = first + (tt - prefix[lo]) * (NT / TERMS);
  w.cnt = min(NT / TERMS, end - w.row0);
  w.b0 = p.nblk * w.split / p.splits;
  w.b1 = p.nblk * (w.split + 1) / p.splits;
  return true;
}

// Byte offset, in its group, of the weight row behind row `i` of a tile. SwiGLU tiles alternate gate and up rows, so that a pair
// sits in neighbouring lanes.
__device__ __forceinline__ uint32_t tile_row(const Params& p, const Item& w, int i) {
  int r;
  if (p.epi & 1) {
    const int half = p.rows >> 1;
    r = min(w.rt * 64 + (i >> 1), half - 1) + (i & 1) * half;
  } else {
    r = min(w.rt * BM + i, p.rows - 1);
  }
  return (uint32_t)r * (uint32_t)p.rb;
}
__device__ __forceinline__ const uint8_t* group_base(const Params& p, const Item& w) { return p.W + (long long)w.group * p.rows * p.rb; }

__device__ __forceinline__ uint32_t mul2(uint32_t x, __half2 s, __half2 off) {
  const __half2 r = __hfma2(*reinterpret_cast<__half2*>(&x), s, off);
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void st_shared4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ float ld_half(const uint8_t* p) { return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short*>(p)))); }

// A decode warp owns RW rows of the tile: it copies their blocks, kSlots - 1 ahead, into a ring of its own (`cp.async`, neighbouring
// lanes take neighbouring bytes: a load of every lane from a row of its own is an L1 pass per row) and decodes from there; a lane
// decodes half a slab of one row at a time.
__device__ __forceinline__ uint32_t ld_shared(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_shared4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}

template <int TYPE> struct Dec;
// A codebook entry per eight weights is read from a random place in shared memory, which with the instructions sets the pace of this type.
// Few instructions per weight: codebook bytes become halves 1024 + v by one byte permutation a
// pair, sign bits reach the tops of the halves by a multiplication, and scale and bias are one fused multiply-add.
template <> struct Dec<T_IQ2_XXS> {
  // a block of 66 bytes starts on 4 bytes or two behind: 17 words hold it
  static constexpr int kCopy = 4, kData = 68, kPitch = 68;
  __device__ static void stage(uint32_t src, int mis, uint32_t dst, int row7, int h, int s, uint32_t grid) {
    const uint32_t a = src + ((mis + 2 + (2 * s + h) * 8) & ~3);
    uint32_t w0 = ld_shared(a), w1 = ld_shared(a + 4);
    if (!mis) {
      const uint32_t w2 = ld_shared(a + 8);
      w0 = __byte_perm(w0, w1, 0x5432);
      w1 = __byte_perm(w1, w2, 0x5432);
    }
    // the odd scale 2 s + 1 as a half, from 1024 + it
    const uint32_t lsw = 0x64016401u + (w1 >> 28) * 0x00020002u;
    const __half2 s2 = __hadd2(*reinterpret_cast<const __half2*>(&lsw), __float2half2_rn(-1024.f)), o2 = __hmul2(s2, __float2half2_rn(-1024.f));
    const uint32_t at = dst | (((4 * h) ^ row7) << 4);
    uint32_t e[4][2];      // all four entries are on their way before the first is used
#pragma unroll
    for (int g = 0; g < 4; ++g)
      asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(e[g][0]), "=r"(e[g][1]) : "r"(grid + ((w0 >> (8 * g)) & 255u) * 8u));
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint32_t lo = e[g][0], hi = e[g][1];
      uint32_t sg = (w1 >> (7 * g)) & 127u;
      sg += (__popc(sg) & 1u) * 128u;                 // the eighth sign makes their number even
      uint32_t x0 = mul2(__byte_perm(lo, 0x64646464u, 0x4240), s2, o2), x1 = mul2(__byte_perm(lo, 0x64646464u, 0x4341), s2, o2);
      uint32_t x2 = mul2(__byte_perm(hi, 0x64646464u, 0x4240), s2, o2), x3 = mul2(__byte_perm(hi, 0x64646464u, 0x4341), s2, o2);
      x0 ^= (sg * ((1u << 15) + (1u << 29))) & 0x80008000u;
      x1 ^= (sg * ((1u << 14) + (1u << 28))) & 0x80008000u;
      x2 ^= (sg * ((1u << 11) + (1u << 25))) & 0x80008000u;
      x3 ^= (sg * ((1u << 10) + (1u << 24))) & 0x80008000u;
      st_shared4(at ^ (g << 4), x0, x1, x2, x3);
    }
  }
};

// scale (m = 0) or minimum (m = 1) of sub-block j from the twelve bytes of a K-quant's 6-bit pairs
__device__ __forceinline__ uint32_t k4_field(const uint32_t (&s)[3], int j, int m) {
  const int k = (j & 3) * 8;
  if (j < 4) return (s[m] >> k) & 63u;
  return ((s[2] >> (k + 4 * m)) & 15u) | (((s[m] >> (k + 6)) & 3u) << 4);
}

// K-quants: low and high nibbles of bytes [16 h, 16 h + 16) of a stage's codes belong to two sub-blocks.
template <int TYPE> struct DecK {
  static constexpr int kCopy = 16, kData = Fmt<TYPE>::bytes, kPitch = Fmt<TYPE>::bytes;
  __device__ static void stage(uint32_t src, int, uint32_t dst, int row7, int h, int st, uint32_t) {
    const uint4 f = ld_shared4(src);
    const uint32_t s[3] = {f.y, f.z, f.w};
    if (st == 4) {      // the codes of the eight minima, for the sums' first (h = 0) and second terms
      uint32_t x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __half2 v = __halves2half2(__uint2half_rn(k4_field(s, 2 * i, 1)), __uint2half_rn(k4_field(s, 2 * i + 1, 1)));
        x[i] = *reinterpret_cast<const uint32_t*>(&v);
      }
      st_shared4(dst + ((h ^ row7) << 4), x[0], x[1], x[2], x[3]);
      return;
    }
    const uint32_t c0 = k4_field(s, 2 * st, 0), c1 = k4_field(s, 2 * st + 1, 0);
    const __half2 s0 = __half2half2(__uint2half_rn(c0)), o0 = __half2half2(__int2half_rn(-1024 * (int)c0));
    const __half2 s1 = __half2half2(__uint2half_rn(c1)), o1 = __half2half2(__int2half_rn(-64 * (int)c1));
    const uint4 q = ld_shared4(src + (TYPE == T_Q5_K ? 48 : 16) + 32 * st + 16 * h);
    const uint4 qh = TYPE == T_Q5_K ? ld_shared4(src + 16 + 16 * h) : make_uint4(0, 0, 0, 0);
    const uint32_t qw[4] = {q.x, q.y, q.z, q.w}, hw[4] = {qh.x, qh.y, qh.z, qh.w};
    uint32_t lo[8], hi[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t w = qw[i], w8 = w >> 8;
      uint32_t a0 = (w & 0x000f000fu) | 0x64006400u, a1 = (w8 & 0x000f000fu) | 0x64006400u;      // 1024 + code
      uint32_t b0 = (w & 0x00f000f0u) | 0x54005400u, b1 = (w8 & 0x00f000f0u) | 0x54005400u;      // 64 + code
      if constexpr (TYPE == T_Q5_K) {
        const uint32_t t = hw[i] >> (2 * st), t8 = t >> 8;      // bit 0: low sub-block, bit 1: high
        a0 |= (t << 4) & 0x00100010u;
        a1 |= (t8 << 4) & 0x00100010u;
        b0 |= (t << 7) & 0x01000100u;
        b1 |= (t8 << 7) & 0x01000100u;
      }
      lo[2 * i] = mul2(a0, s0, o0);
      lo[2 * i + 1] = mul2(a1, s0, o0);
      hi[2 * i] = mul2(b0, s1, o1);
      hi[2 * i + 1] = mul2(b1, s1, o1);
    }
    st_shared4(dst + (((2 * h) ^ row7) << 4), lo[0], lo[1], lo[2], lo[3]);
    st_shared4(dst + (((2 * h + 1) ^ row7) << 4), lo[4], lo[5], lo[6], lo[7]);
    st_shared4(dst + (((4 + 2 * h) ^ row7) << 4), hi[0], hi[1], hi[2], hi[3]);
    st_shared4(dst + (((5 + 2 * h) ^ row7) << 4), hi[4], hi[5], hi[6], hi[7]);
  }
};
template <> struct Dec<T_Q4_K> : DecK<T_Q4_K> {};
template <> struct Dec<T_Q5_K> : DecK<T_Q5_K> {};

// E4M3 codes are fp16 numbers already; the rows of the ring are 16 bytes apart from whole lines (bank conflicts).
template <> struct Dec<T_E4M3> {
  static constexpr int kCopy = 16, kData = 128, kPitch = 144;
  __device__ static void stage(uint32_t src, int, uint32_t dst, int row7, int h, int s, uint32_t) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint4 v = ld_shared4(src + 64 * s + 32 * h + 16 * i);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      uint32_t x[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[j] & 0xffffu), __NV_E4M3);
        const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[j] >> 16), __NV_E4M3);
        x[2 * j] = (uint32_t)lo.x | (uint32_t)lo.y << 16;
        x[2 * j + 1] = (uint32_t)hi.x | (uint32_t)hi.y << 16;
      }
      st_shared4(dst + (((4 * h + 2 * i) ^ row7) << 4), x[0], x[1], x[2], x[3]);
      st_shared4(dst + (((4 * h + 2 * i + 1) ^ row7) << 4), x[4], x[5], x[6], x[7]);
    }
  }
};

__host__ __device__ constexpr uint32_t tmem_columns(uint32_t n) {
  uint32_t c = 32;
  while (c < n) c *= 2;
  return c;
}

// By one thread, behind the CTA's stores of its part: *last says whether the other parts are there.
__device__ __forceinline__ void count_part(const Params& p, const Item& w, uint32_t* last) {
  const uint32_t n = atomicAdd(p.counters + w.tile, 1u);
  *last = n == (uint32_t)p.splits - 1u;
  if (*last) p.counters[w.tile] = 0u;
  __threadfence();
}

template <int WARPS>
__device__ __forceinline__ void fold_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory");
}

// The rest of a fold warp's items, from `i` on, after a wait that ran out: NaN in their places, so that the result cannot be taken
// for one, and every part counted, so that the counters are back at zero when the launch is over. Kept out of the loop that it ends.
template <int NT, int TERMS, int WARPS>
__device__ __noinline__ void give_up(const Params& p, const int* prefix, int row_tiles, int i, int c0, uint32_t* shared_last) {
  const int tid = threadIdx.x, lr = ((tid >> 5) & 3) * 32 + (tid & 31), cols = WARPS == 8 ? NT / 2 : NT;
  const float nan = __uint_as_float(0x7fffffffu);
  Item w;
  for (; item_at<NT, TERMS>(p, prefix, row_tiles, i, w); i += gridDim.x) {
    if (p.splits > 1) {
      float* part = p.ws + ((size_t)w.tile * p.splits + w.split) * NT * BM + lr;
      for (int c = c0; c < c0 + cols; ++c) __stcg(part + (size_t)c * BM, nan);
      __threadfence();
      fold_sync<WARPS>();
      if (tid == 0) count_part(p, w, shared_last);
      fold_sync<WARPS>();
      const uint32_t last = *(volatile uint32_t*)shared_last;
      fold_sync<WARPS>();
      if (!last) continue;
    }
    const bool glu = p.epi & 1;
    const int n = glu ? w.rt * 64 + (lr >> 1) : w.rt * BM + lr;
    if (n >= (glu ? p.rows >> 1 : p.rows)) continue;
    for (int m = c0 / TERMS; m < min(w.cnt, (c0 + cols) / TERMS); ++m) {
      const size_t at = (size_t)(w.row0 + m) * p.ldo + n;
      if (p.epi == OUT_F32 || p.epi == OUT_SWIGLU_F32) ((float*)p.out)[at] = nan;
      else ((bf16*)p.out)[at] = __float2bfloat16(nan);
    }
  }
}

template <int TYPE, int NT, int TERMS>
__global__ void __launch_bounds__(Shape<TYPE, NT>::kThreads, Shape<TYPE, NT>::kCtas)
quant_umma_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ Params p) {
  using S = Shape<TYPE, NT>;
  constexpr int kStages = S::kStages, BB = Fmt<TYPE>::bytes;
  constexpr bool MINS = Fmt<TYPE>::mins;
  constexpr int ST = MINS ? 3 : Fmt<TYPE>::k / 128;      // stages of a block; the third one has the minima in its first 16 places
  constexpr uint32_t kBufCols = MINS ? 2 * NT : NT;
  // One CTA can have several parts of K where a decode step uses it (16 columns; wider tiles have no registers for it): columns of
  // their sum, behind the two accumulators.
  constexpr bool kParts = TYPE != T_E4M3 && NT == 16;
  constexpr uint32_t kSums = 2 * kBufCols, kTmemCols = tmem_columns(kSums + (kParts ? NT : 0));
  extern __shared__ uint8_t smem_raw[];
  using D = Dec<TYPE>;
  using Sm = Smem<S, D::kPitch>;
  Sm& sm = *reinterpret_cast<Sm*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row_tiles = (p.epi & 1) ? ((p.rows >> 1) + 63) / 64 : (p.rows + BM - 1) / BM;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sm.full[s], S::kDecWarps + 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.acc_full[b], 1);
      mbar_init(&sm.acc_empty[b], S::kFoldWarps);
    }
    mbar_init(&sm.drained, 1);
    sm.abort_flag = 0;
    mbar_fence_init();
  }
  for (int g = tid; g < p.n_groups; g += S::kThreads) {
    const int n = p.seg ? max(p.seg[g + 1] - p.seg[g], 0) : p.M;
    sm.prefix[g] = (n + NT / TERMS - 1) / (NT / TERMS);
  }
  __syncthreads();
  if (warp == 1) {
    // token tiles before each group, 32 groups at a time
    int run = 0;
    for (int g0 = 0; g0 < p.n_groups; g0 += 32) {
      const int g = g0 + lane;
      const int n = g < p.n_groups ? sm.prefix[g] : 0;
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (g < p.n_groups) sm.prefix[g] = run + inc - n;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) sm.prefix[p.n_groups] = run;
  }
  if (warp == 2) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  if constexpr (TYPE == T_IQ2_XXS)
    for (int i = tid; i < 256; i += S::kThreads) sm.grid[i] = kIq2xxsGrid[i];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;

  if (warp < S::kFoldWarps) {
    // ---------------- fold and epilogue ----------------
    const int q = warp & 3, c0 = (warp >> 2) * S::kFoldCols, lr = q * 32 + lane;
    uint32_t blk = 0;
    Item w;
    bool ok = true;
    // an earlier product of the step gave up: this one does as if its first wait had
    const bool dead = p.status != nullptr && __any_sync(0xffffffffu, *(const volatile uint32_t*)p.status);
    if (dead) sm.abort_flag = 1u;
    for (int i = blockIdx.x; ok && item_at<NT, TERMS>(p, sm.prefix, row_tiles, i, w); i += gridDim.x) {
      const uint8_t* row = group_base(p, w) + tile_row(p, w, lr);
      float acc[S::kFoldCols];
#pragma unroll
      for (int c = 0; c < S::kFoldCols; ++c) acc[c] = 0.f;
      const float* ws = nullptr;
      if constexpr (TYPE == T_E4M3) {
        const int half = p.rows >> 1;
        const int r = (p.epi & 1) ? min(w.rt * 64 + (lr >> 1), half - 1) + (lr & 1) * half : w.rt * BM;
        ws = p.w_scale + (size_t)(r >> 7) * p.w_ld;
      }
      auto factor = [&](int b) { return TYPE == T_E4M3 ? __ldg(ws + b) : ld_half(row + b * BB); };
      float d = factor(w.b0), dm = MINS ? ld_half(row + w.b0 * BB + 2) : 0.f;
      [[maybe_unused]] int part = 0, part_end = kParts && p.splits == 1 && p.parts > 1 ? p.nblk / p.parts : -1;
      for (int b = w.b0; b < w.b1; ++b, ++blk) {
        const int nb = min(b + 1, p.nblk - 1);
        const float dn = factor(nb), dmn = MINS ? ld_half(row + nb * BB + 2) : 0.f;
        const int buf = blk & 1;
        if (dead || !mbar_wait_uniform(&sm.acc_full[buf], (blk >> 1) & 1, &sm.abort_flag, p.status, 31)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const float f = TYPE == T_IQ2_XXS ? 0.125f * d : d;
        const uint32_t t = tmem_base + buf * kBufCols + c0 + ((uint32_t)(q * 32) << 16);
#pragma unroll
        for (int c = 0; c < S::kFoldCols; c += 16) {
          uint32_t r[16];
          tmem_ld_32x16(t + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(f, __uint_as_float(r[j]), acc[c + j]);
          if constexpr (MINS) {
            tmem_ld_32x16(t + NT + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(-dm, __uint_as_float(r[j]), acc[c + j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acc_empty[buf]);
        d = dn;
        dm = dmn;
        if constexpr (kParts)
          if (b + 1 == part_end) {
            const uint32_t ts = tmem_base + kSums + ((uint32_t)(q * 32) << 16);
            uint32_t r[16] = {};
            if (part > 0) {
              tmem_ld_32x16(ts, r);
              tmem_ld_wait();
            }
            const bool more = b + 1 < w.b1;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              acc[j] += __uint_as_float(r[j]);
              r[j] = __float_as_uint(acc[j]);
              if (more) acc[j] = 0.f;
            }
            if (more) {
              tmem_st_32x16(ts, r);
              tmem_st_wait();
            }
            ++part;
            part_end = p.nblk * (part + 1) / p.parts;
          }
      }
      if (!ok) {
        give_up<NT, TERMS, S::kFoldWarps>(p, sm.prefix, row_tiles, i, c0, &sm.last);
        break;
      }
      if (p.splits > 1) {
        float* part = p.ws + ((size_t)w.tile * p.splits + w.split) * NT * BM + lr;
#pragma unroll
        for (int c = 0; c < S::kFoldCols; ++c) __stcg(part + (size_t)(c0 + c) * BM, acc[c]);
        __threadfence();
        fold_sync<S::kFoldWarps>();
        if (tid == 0) count_part(p, w, &sm.last);
        fold_sync<S::kFoldWarps>();
        const uint32_t last = sm.last;
        fold_sync<S::kFoldWarps>();
        if (!last) continue;
        __threadfence();
        const float* all = p.ws + (size_t)w.tile * p.splits * NT * BM + lr;
#pragma unroll
        for (int c = 0; c < S::kFoldCols; ++c) acc[c] = 0.f;
        for (int s = 0; s < p.splits; ++s)
#pragma unroll
          for (int c = 0; c < S::kFoldCols; ++c) acc[c] += __ldcg(all + ((size_t)s * NT + c0 + c) * BM);
      }
      // columns of a token row next to one another
      constexpr int kRows = S::kFoldCols / TERMS;
      float v[kRows];
#pragma unroll
      for (int m = 0; m < kRows; ++m) v[m] = TERMS == 2 ? acc[2 * m] + acc[2 * m + 1] : acc[m];
      const int m0 = c0 / TERMS;
#pragma unroll
      for (int m = 0; m < kRows; ++m)
        if (m0 + m < w.cnt) v[m] *= __ldg(p.row_scale + w.row0 + m0 + m);
      if (p.epi & 1) {
        // gate and up of an output sit in a pair of lanes, of which each takes every second token row
        const int j = w.rt * 64 + (lr >> 1);
        const bool up = lane & 1, in = j < (p.rows >> 1);
#pragma unroll
        for (int m = 0; m < kRows; m += 2) {
          const float got = __shfl_xor_sync(0xffffffffu, up ? v[m] : v[m + 1], 1);
          float g = up ? got : v[m], u = up ? v[m + 1] : got;
          if (p.limit > 0.f) {
            g = fminf(g, p.limit);
            u = fminf(fmaxf(u, -p.limit), p.limit);
          }
          const int mm = m0 + m + (up ? 1 : 0);
          if (in && mm < w.cnt) {
            const size_t at = (size_t)(w.row0 + mm) * p.ldo + j;
            if (p.epi == OUT_SWIGLU_F32) ((float*)p.out)[at] = silu(g) * u;
            else ((bf16*)p.out)[at] = __float2bfloat16(silu(g) * u);
          }
        }
      } else {
        const int n = w.rt * BM + lr;
        if (n < p.rows) {
#pragma unroll
          for (int m = 0; m < kRows; ++m) {
            if (m0 + m >= w.cnt) break;
            const size_t at = (size_t)(w.row0 + m0 + m) * p.ldo + n;
            if (p.epi == OUT_F32) ((float*)p.out)[at] = v[m];
            else if (p.epi == OUT_RESID) ((bf16*)p.out)[at] = __float2bfloat16(v[m] + __bfloat162float(p.resid[at]));
            else ((bf16*)p.out)[at] = __float2bfloat16(v[m]);
          }
        }
      }
    }
  } else if (warp == S::kFoldWarps) {
    // ---------------- MMA issuer ----------------
    // The whole warp walks the loop and one lane issues: addresses and descriptors are then uniform, which is what the
    // instructions take; computed by a lone lane they cost more than the products.
    constexpr uint32_t idesc = umma_idesc(0, 0, BM, NT);
    const uint64_t da0 = smem_desc_k_sw128(smem_u32(sm.a[0])), db0 = smem_desc_k_sw128(smem_u32(sm.b[0]));
    const bool leader = elect_one();
    uint32_t st = 0, ph = 0, blk = 0;
    Item w;
    bool ok = true;
    for (int i = blockIdx.x; ok && item_at<NT, TERMS>(p, sm.prefix, row_tiles, i, w); i += gridDim.x) {
      for (int b = w.b0; ok && b < w.b1; ++b, ++blk) {
        const int buf = blk & 1;
        if (!mbar_wait_uniform(&sm.acc_empty[buf], ((blk >> 1) & 1) ^ 1, &sm.abort_flag, p.status, 32)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t acc = tmem_base + buf * kBufCols;
#pragma unroll 1
        for (int s = 0; s < ST; ++s) {
          if (!mbar_wait_uniform(&sm.full[st], ph, &sm.abort_flag, p.status, 33)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t da = da0 + st * (S::kABytes >> 4), db = db0 + st * (S::kBBytes >> 4);
          if (leader) {
            if (s < 2) {
#pragma unroll
              for (int k = 0; k < 8; ++k)
                umma_f16(acc, da + (k >> 2) * (BM * 128 >> 4) + (k & 3) * 2, db + (k >> 2) * (NT * 128 >> 4) + (k & 3) * 2, idesc, (s > 0 || k > 0) ? 1u : 0u);
            } else {
              umma_f16(acc + NT, da, db, idesc, 0u);
            }
            umma_commit(&sm.empty[st]);
            if (s == ST - 1) umma_commit(&sm.acc_full[buf]);
          }
          __syncwarp();
          if (++st == kStages) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    }
    if (!ok) {
      // gave up: the products in flight end before their tensor memory is freed
      if (leader) umma_commit(&sm.drained);
      __syncwarp();
      for (uint32_t n = 0; n < kDrainPolls && !mbar_try_wait(&sm.drained, 0); ++n) {}
    }
  } else if (warp == S::kFoldWarps + 1) {
    // ---------------- token tiles ----------------
    if (lane == 0) {
      tma_prefetch_desc(&tmap);
      uint32_t st = 0, ph = 1, issued = 0;
      Item w;
      bool ok = true;
      for (int i = blockIdx.x; ok && item_at<NT, TERMS>(p, sm.prefix, row_tiles, i, w); i += gridDim.x)
        for (int x = w.b0 * Fmt<TYPE>::cols; ok && x < w.b1 * Fmt<TYPE>::cols;) {
#pragma unroll
          for (int s = 0; s < ST; ++s, ++issued) {
            if (!mbar_wait(&sm.empty[st], ph, &sm.abort_flag, p.status, 35)) {
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&sm.full[st], (s < 2 ? 2 : 1) * NT * 128);
            tma_load_2d(sm.b[st], &tmap, &sm.full[st], x, w.row0 * TERMS);
            x += 64;
            if (s < 2) {
              tma_load_2d(sm.b[st] + NT * 128, &tmap, &sm.full[st], x, w.row0 * TERMS);
              x += 64;
            }
            if (++st == kStages) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
      if (sm.abort_flag) {
        // gave up: copies in flight land before the CTA exits
        for (uint32_t j = issued > (uint32_t)kStages ? issued - kStages : 0; j < issued; ++j)
          for (uint32_t n = 0; n < kDrainPolls; ++n)
            if (mbar_try_wait(&sm.full[j % kStages], (j / kStages) & 1)) break;
      }
    }
  } else {
    // ---------------- decode ----------------
    constexpr int RW = S::kRows, SB = 16 / RW;            // rows of a warp; slabs of a stage that it decodes side by side
    constexpr int kRowChunks = D::kData / D::kCopy, kChunks = RW * kRowChunks;      // copies of a block of a row, of the warp's rows
    constexpr int kCopies = (kChunks + 31) / 32;
    const int dw = warp - S::kFoldWarps - 2, r = lane % RW, lr = dw * RW + r, h = (lane / RW) & 1, sb = lane / (2 * RW);
    const uint32_t ring = smem_u32(sm.ring[0]) + dw * RW * D::kPitch;
    // The copy cursor runs kSlots - 1 blocks ahead of the decoding, over the ends of the CTA's items.
    int ci = blockIdx.x, cb = 0, cb1 = 0;
    uint32_t slot_fill = 0;
    bool more = true;
    const uint8_t* base = nullptr;
    uint32_t off[kCopies];
    auto copy_next = [&]() {
      if (more && cb == cb1) {
        Item c;
        more = item_at<NT, TERMS>(p, sm.prefix, row_tiles, ci, c);
        ci += gridDim.x;
        if (more) {
          base = group_base(p, c);
          cb = c.b0;
          cb1 = c.b1;
#pragma unroll
          for (int k = 0; k < kCopies; ++k) {
            const int n = min(lane + 32 * k, kChunks - 1), j = n / kRowChunks;
            off[k] = tile_row(p, c, dw * RW + j) + (n - j * kRowChunks) * D::kCopy;
          }
        }
      }
      if (more) {
#pragma unroll
        for (int k = 0; k < kCopies; ++k) {
          uint32_t o = off[k] + (uint32_t)cb * BB;
          if constexpr (D::kCopy == 4) o &= ~3u;
          const int n = lane + 32 * k, j = n / kRowChunks;
          const uint32_t dst = ring + slot_fill * (BM * D::kPitch) + (D::kData == D::kPitch ? n * D::kCopy : j * D::kPitch + (n - j * kRowChunks) * D::kCopy);
          if ((k + 1) * 32 <= kChunks || n < kChunks) {
            if constexpr (D::kCopy == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(base + o) : "memory");
            else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(base + o) : "memory");
          }
        }
        ++cb;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      slot_fill = slot_fill + 1 == S::kSlots ? 0 : slot_fill + 1;
    };
#pragma unroll
    for (int k = 0; k + 1 < S::kSlots; ++k) copy_next();
    const uint32_t grid = smem_u32(sm.grid);
    uint32_t st = 0, ph = 1, slot = 0;
    Item w;
    bool ok = true;
    for (int i = blockIdx.x; ok && item_at<NT, TERMS>(p, sm.prefix, row_tiles, i, w); i += gridDim.x) {
      const uint32_t own = tile_row(p, w, lr);
      for (int b = w.b0; ok && b < w.b1; ++b) {
        __syncwarp();       // the slot that is filled now has been read by all lanes
        copy_next();
        asm volatile("cp.async.wait_group %0;" ::"n"(S::kSlots - 1) : "memory");
        __syncwarp();       // every lane's copies of this block are there
        const uint32_t src = ring + slot * (BM * D::kPitch) + r * D::kPitch;
        slot = slot + 1 == S::kSlots ? 0 : slot + 1;
        const int mis = D::kCopy == 4 ? (int)((own + (uint32_t)b * BB) & 2u) : 0;
#pragma unroll 1      // code that fits the instruction caches
        for (int s = 0; s < ST; ++s) {
          if (!mbar_wait_uniform(&sm.empty[st], ph, &sm.abort_flag, p.status, 36)) {
            ok = false;
            break;
          }
          const uint32_t dst = smem_u32(sm.a[st]) + lr * 128;
          if (s < 2) {       // two slabs of 64
#pragma unroll 1
            for (int e = 0; e < 2; e += SB) {
              const int slab = SB == 2 ? sb : e;
              D::stage(src, mis, dst + slab * (BM * 128), lr & 7, h, 2 * s + slab, grid);
            }
          } else if (sb == 0) {
            D::stage(src, mis, dst, lr & 7, h, 4, grid);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.full[st]);
          if (++st == kStages) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Token rows for the product: fp16 under a power of two per row (1024 at most, so that a bf16 value within 2^-24 of the row's
// largest keeps all its bits), in one or two terms (22 to 23 bits of an fp32 value), in the order of the decoded weights; with `mins` the sums over every 32
// values follow each 256. One block per row.
struct StageParams {
  const void* x;
  int x_f32, ldx, K;
  const int* index;       // row gather; null: identity
  const float* gamma;     // RMSNorm with its result rounded to bf16; null: none
  float eps;
  int plus_one;           // the norm multiplies by 1 + gamma
  const float* add;       // [rows, K] added to x first, the sum rounded to bf16 and written to `sum` (not with index)
  bf16* sum;
  bf16* norm;             // the normed rows [rows, K] as well; null: not kept
  int terms, mins, natural;
  __half* out;
  float* row_scale;
  uint32_t* counters;
  int n_counters;
};

__global__ void __launch_bounds__(1024) quant_stage_rows_kernel(const StageParams p) {
  extern __shared__ __align__(16) float xs[];      // [K]
  __shared__ float red[40];
  const int r = blockIdx.x, tid = threadIdx.x, stride = blockDim.x * 4;
  if (r == 0)
    for (int i = tid; i < p.n_counters; i += blockDim.x) p.counters[i] = 0u;
  const long long src = p.index ? p.index[r] : r;
  float ss = 0.f, mx = 0.f;
  for (int k = tid * 4; k < p.K; k += stride) {
    float4 v;
    if (p.x_f32) {
      v = *reinterpret_cast<const float4*>((const float*)p.x + src * p.ldx + k);
    } else {
      const uint2 u = *reinterpret_cast<const uint2*>((const bf16*)p.x + src * p.ldx + k);
      v = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    }
    if (p.add != nullptr) {
      const float4 a = *reinterpret_cast<const float4*>(p.add + src * p.K + k);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x + a.x, v.y + a.y), hi = __floats2bfloat162_rn(v.z + a.z, v.w + a.w);
      const uint2 u = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      *reinterpret_cast<uint2*>(p.sum + src * p.ldx + k) = u;
      v = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    }
    *reinterpret_cast<float4*>(xs + k) = v;
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
  }
  if (p.gamma != nullptr) {
    const float rs = rsqrtf(block_sum(ss, red) / (float)p.K + p.eps);
    mx = 0.f;
    for (int k = tid * 4; k < p.K; k += stride) {
      float4 v = *reinterpret_cast<const float4*>(xs + k);
      float4 g = *reinterpret_cast<const float4*>(p.gamma + k);
      if (p.plus_one) g = make_float4(1.f + g.x, 1.f + g.y, 1.f + g.z, 1.f + g.w);
      v.x = __bfloat162float(__float2bfloat16(v.x * rs * g.x));
      v.y = __bfloat162float(__float2bfloat16(v.y * rs * g.y));
      v.z = __bfloat162float(__float2bfloat16(v.z * rs * g.z));
      v.w = __bfloat162float(__float2bfloat16(v.w * rs * g.w));
      *reinterpret_cast<float4*>(xs + k) = v;
      if (p.norm != nullptr) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
        *reinterpret_cast<uint2*>(p.norm + (size_t)r * p.K + k) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
      mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    }
  }
  mx = block_max(mx, red);
  // up = 2^e with mx * up in [512, 1024); rows of zeros, infinities or NaN stay as they are
  const int ex = (int)(__float_as_uint(mx) >> 23);
  const int e = (ex == 0 || ex >= 255) ? 0 : min(126, 9 - (ex - 127));
  const float up = __uint_as_float((uint32_t)(127 + e) << 23), down = ldexpf(1.f, -e);
  if (tid == 0) p.row_scale[r] = down;
  const int pitch = p.mins ? (p.K >> 8) * 320 : p.K;
  __half* out = p.out + (size_t)r * p.terms * pitch;
  for (int k = tid * 4; k < p.K; k += stride) {      // K is a multiple of 128: whole warps
    const float4 v = *reinterpret_cast<const float4*>(xs + k);
    const float a[4] = {v.x * up, (p.natural ? v.y : v.z) * up, (p.natural ? v.z : v.y) * up, v.w * up};
    const int at = p.mins ? (k >> 8) * 320 + (k & 255) : k;
    __half2 h0 = __floats2half2_rn(a[0], a[1]), h1 = __floats2half2_rn(a[2], a[3]);
    *reinterpret_cast<uint2*>(out + at) = make_uint2(*reinterpret_cast<uint32_t*>(&h0), *reinterpret_cast<uint32_t*>(&h1));
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    float s = (f0.x + f0.y) + (f1.x + f1.y);
    if (p.terms == 2) {
      const __half2 l0 = __floats2half2_rn(a[0] - f0.x, a[1] - f0.y), l1 = __floats2half2_rn(a[2] - f1.x, a[3] - f1.y);
      *reinterpret_cast<uint2*>(out + pitch + at) = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
      const float2 g0 = __half22float2(l0), g1 = __half22float2(l1);
      s += (g0.x + g0.y) + (g1.x + g1.y);
    }
    if (p.mins) {      // sums of the values as they are multiplied: a block's codes and minima nearly cancel
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if ((tid & 7) == 0) {
        __half* m = out + (k >> 8) * 320 + 256 + ((k & 255) >> 5);
        const __half hi = __float2half_rn(s);
        m[0] = hi;
        m[8] = __float2half_rn(s - __half2float(hi));
        if (p.terms == 2) {       // the second row holds the rest of the values: its sums are part of the first one's
          m[pitch] = __float2half_rn(0.f);
          m[pitch + 8] = __float2half_rn(0.f);
        }
      }
    }
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

template <int TYPE, int NT, int TERMS>
int launch(const void* staged, int total_rows, const Params& p, int sms, cudaStream_t stream) {
  EncodeTiledFn encode = encode_fn();
  if (encode == nullptr) return PK_ERR_UNSUPPORTED;
  CUtensorMap map;
  const cuuint64_t pitch = (cuuint64_t)p.nblk * Fmt<TYPE>::cols;
  const cuuint64_t gdim[2] = {pitch, (cuuint64_t)total_rows * TERMS}, gstride[1] = {pitch * 2};
  const cuuint32_t box[2] = {64, NT}, estr[2] = {1, 1};
  if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(staged), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return PK_ERR_CUDA;
  const size_t smem = sizeof(Smem<Shape<TYPE, NT>, Dec<TYPE>::kPitch>) + 1024;
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(quant_umma_kernel<TYPE, NT, TERMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  quant_umma_kernel<TYPE, NT, TERMS><<<sms * Shape<TYPE, NT>::kCtas, Shape<TYPE, NT>::kThreads, smem, stream>>>(map, p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

template <int TYPE>
int launch_shape(int nt, int terms, const void* staged, int total_rows, const Params& p, int sms, cudaStream_t stream) {
  if (terms == 1) {
    if (nt == 16) return launch<TYPE, 16, 1>(staged, total_rows, p, sms, stream);
    if (nt == 32) return launch<TYPE, 32, 1>(staged, total_rows, p, sms, stream);
    return launch<TYPE, 64, 1>(staged, total_rows, p, sms, stream);
  }
  if (nt == 16) return launch<TYPE, 16, 2>(staged, total_rows, p, sms, stream);
  if (nt == 32) return launch<TYPE, 32, 2>(staged, total_rows, p, sms, stream);
  return launch<TYPE, 64, 2>(staged, total_rows, p, sms, stream);
}

bool has_mins(int type) { return type == T_Q4_K || type == T_Q5_K; }
int type_bytes(int type) { return type == T_IQ2_XXS ? 66 : type == T_Q4_K ? 144 : type == T_Q5_K ? 176 : type == T_E4M3 ? 128 : 0; }
int type_k(int type) { return type == T_E4M3 ? 128 : 256; }

}  // namespace

// fp16 elements of one term of a staged row; 0 when the type has no tensor-core path.
PK_API int pk_quant_stage_pitch(int type, int K) {
  if (type_bytes(type) == 0 || K < 1 || K % type_k(type) != 0) return 0;
  return has_mins(type) ? (K >> 8) * 320 : K;
}

// rows of x (bf16, or fp32 with x_f32; row stride ldx elements, a multiple of four, 16-byte aligned base) -> staged [rows * terms, pitch]
// fp16 and row_scale [rows]. Also zeroes `n_counters` words for the product that follows.
// `add` (fp32 [rows, K], with `sum`: bf16, row stride ldx) is added to x first and the rounded sum kept; `norm` (bf16 [rows, K],
// with gamma) keeps the normed rows.
PK_API int pk_quant_stage_rows(const void* x, int x_f32, int ldx, int K, const int* index, int rows, const float* gamma, float eps, int plus_one,
                               const float* add, void* sum, void* norm, int type, int terms, void* staged, float* row_scale, uint32_t* counters, int n_counters, cudaStream_t stream) {
  if (x == nullptr || staged == nullptr || row_scale == nullptr || rows < 1 || terms < 1 || terms > 2 || pk_quant_stage_pitch(type, K) == 0 || (ldx & 3) != 0 ||
      ((uintptr_t)x & 15) != 0 || ((uintptr_t)staged & 15) != 0 || ((uintptr_t)gamma & 15) != 0 || n_counters < 0 || (n_counters > 0 && counters == nullptr) || (norm != nullptr && (gamma == nullptr || ((uintptr_t)norm & 7) != 0)) || (add != nullptr && (sum == nullptr || index != nullptr || ((uintptr_t)add & 15) != 0)))
    return PK_ERR_BAD_ARG;
  const size_t smem = (size_t)K * sizeof(float);
  if (smem > 200 * 1024) return PK_ERR_UNSUPPORTED;
  if (smem > kPlainSmem) {
    static PkDeviceOnce once;
    if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
      if (cudaFuncSetAttribute(quant_stage_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) {
        pk_set_last_cuda_error((int)cudaGetLastError());
        return PK_ERR_CUDA;
      }
      once_guard.done();
    }
  }
  const StageParams p{x, x_f32, ldx, K, index, gamma, eps, plus_one, add, (pk::bf16*)sum, (pk::bf16*)norm, terms, has_mins(type) ? 1 : 0, type == T_E4M3 ? 1 : 0, (__half*)staged, row_scale, counters, n_counters};
  // a block per row: with few rows a thread per four elements (13 rows of 5120 to 17408: mean 6.2 -> 4.6 us, one of 3072: 3.8 -> 2.9), with many the blocks hide one another
  const int threads = rows <= 148 ? min(1024, (K / 4 + 31) / 32 * 32) : 256;
  quant_stage_rows_kernel<<<rows, threads, smem, stream>>>(p);
  PK_CHECK_LAUNCH();
  return PK_OK;
}

// out[t, n] = row_scale[t] * staged[t] . W[g(t), n]: W [n_groups * N] raw rows of `type`; token rows seg[g] .. seg[g + 1] belong to
// group g (seg null: all `rows` to the one group). epi 0 bf16, 1 SwiGLU bf16, 2 fp32, 3 SwiGLU fp32 (N / 2 gate rows, then as
// many up rows), 4 bf16 with `resid` added. `columns` 16, 32 or 64 of a tile. K is summed in `parts`,
// by as many CTAs (splits = parts) or, with 16 columns, by one (splits 1) to the same bits. splits > 1 needs ws (tiles * splits * columns * 128 floats)
// and one zeroed counter per tile. E4M3 (type 20): W [N, K] codes, w_scale [ceil(N / 128), w_ld] factors of its 128 x 128 blocks;
// 32 or 64 columns (up to 16 rows are rows_fp8.cu's).
PK_API int pk_quant_rows(const void* W, int type, int N, int K, const int* seg, int n_groups, int rows, const void* staged, const float* row_scale,
                         int terms, int epi, void* out, int ldo, const void* resid, float limit, int columns, int parts, int splits, float* ws, uint32_t* counters, uint32_t* status,
                         const float* w_scale, int w_ld, int sm_count, cudaStream_t stream) {
  if (W == nullptr || staged == nullptr || row_scale == nullptr || out == nullptr || rows < 1 || N < 1 || n_groups < 1 || n_groups > kMaxGroups ||
      (seg == nullptr && n_groups != 1) || terms < 1 || terms > 2 || epi < 0 || epi > 4 || (epi == OUT_RESID && resid == nullptr) || ((epi & 1) && (N & 1)) || parts < 1 || (splits != parts && (splits != 1 || columns != 16)) ||
      (splits > 1 && (ws == nullptr || counters == nullptr)) || (columns != 16 && columns != 32 && columns != 64) || pk_quant_stage_pitch(type, K) == 0 ||
      parts > K / type_k(type) || (type == T_E4M3 && (parts != splits || w_scale == nullptr || terms != 1 || n_groups != 1 || columns == 16)) || ((uintptr_t)W & 15) != 0 || ((uintptr_t)staged & 15) != 0)
    return PK_ERR_BAD_ARG;
  const int nblk = K / type_k(type);
  const long long group_bytes = (long long)nblk * type_bytes(type) * N;      // IQ2 blocks are copied by four bytes
  if (group_bytes >= (1ll << 32) || (type == T_IQ2_XXS && (group_bytes & 3) != 0)) return PK_ERR_UNSUPPORTED;
  const Params p{(const uint8_t*)W, (long long)nblk * type_bytes(type), nblk, N, n_groups, seg, rows, epi, limit, out, ldo, (const pk::bf16*)resid, row_scale, w_scale, w_ld,
                 parts, splits, ws, counters, status};
  const int sms = sm_count > 0 ? sm_count : 148;
  if (type == T_IQ2_XXS) return launch_shape<T_IQ2_XXS>(columns, terms, staged, rows, p, sms, stream);
  if (type == T_Q4_K) return launch_shape<T_Q4_K>(columns, terms, staged, rows, p, sms, stream);
  if (type == T_Q5_K) return launch_shape<T_Q5_K>(columns, terms, staged, rows, p, sms, stream);
  if (columns == 32) return launch<T_E4M3, 32, 1>(staged, rows, p, sms, stream);
  return launch<T_E4M3, 64, 1>(staged, rows, p, sms, stream);
}
