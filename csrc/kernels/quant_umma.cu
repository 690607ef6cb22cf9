// Products of few token rows with quantised weights through the 5th-generation tensor cores: linear layers and routed experts on raw
// GGUF blocks, linear layers in E4M3 with a scale per 128 x 128 block.
//
// The weights are the M side of the product: a tile is 128 weight rows times up to 64 token columns (a token row takes one, or two where its
// values are two terms), so that a step with one token decodes every weight once and one with hundreds once per 64 columns; none is
// expanded in HBM. Decode warps write the INTEGER part of the weights (codebook entry or code times the sub-block's scale: at most 11 bits)
// as fp16 into tensor memory, from where the products take their A operand: shared memory then holds the raw blocks, the token columns
// and the lookups only. Token rows are fp16 under a power of two per row (`pk_quant_stage_rows`), and the fp32 factor of a block is
// applied when the block's accumulator is folded from TMEM into registers: every product of a bf16 value within 2^-24 of its row's
// largest is exact (smaller ones lose bits that fp16 has no place for) and every sum is fp32. K-quants carry a minimum per 32 weights:
// these are a second, 16-wide product per block, of the minima's codes with the sums of the token values (two fp16 terms each).
//
// Measured, 256 experts of the MiniMax-M2 shape in IQ2_XXS, gate and up / down, us (before: weights through swizzled shared memory, entries
// of 8 bytes from one copy of the codebook, whose bank conflicts and the stores kept the shared-memory pipe 77 % busy): 184 routes
// 410 / 223 -> 215 / 127, 2048 routes 815 / 432 -> 414 / 223, 12000 routes 957 / 510 -> 559 / 289. Bound by the instructions of the decode:
// 4330 warp instructions per 32768 weights, of which 2450 turn codes into halves; issue slots 75 %, ALU 67 %, shared-memory pipe 35 %. Of
// Q5_K, 256 rows of 8192 x 3072: 62 -> 43; E4M3, 40 rows of 34816 x 5120: 68 -> 57.
//
//   warps 0-3 (0-7 for 64 columns)  fold: TMEM -> fp32 registers with the block factors, epilogue
//   next warp                       MMA issuer
//   next warp                       token tiles, and raw blocks whose rows are whole 16 bytes, by TMA (no multicast)
//   next 2 warps                    raw blocks of IQ2_XXS, by cp.async
//   16 warps                        decode
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
constexpr int kMaxTiles = 1024;      // of token rows whose group and place are looked up
constexpr int kIq2Table = (256 + 128) * 32;      // words: codes of the codebook's entries, then sign patterns, each once per lane
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
  int row_tiles;
  int step_split, step_rt, step_tt;      // from an item of a CTA to its next one
};

// One CTA per SM. A unit is 256 weights of every row of a tile (a GGUF block, two E4M3 blocks), in four pieces of 64.
template <int TYPE, int NT>
struct Shape {
  static constexpr int kFoldWarps = NT == 64 ? 8 : 4;
  static constexpr int kFoldCols = NT == 64 ? 32 : NT;
  static constexpr int kDecWarps = 16;                          // four of each quarter of the rows: one per piece
  static constexpr int kSlots = TYPE == T_IQ2_XXS ? (NT == 64 ? 6 : 8) : TYPE == T_E4M3 ? 4 : 5;      // units of raw blocks
  static constexpr int kBBytes = NT * 128;                      // token columns of a piece
  static constexpr int kThreads = 32 * (kFoldWarps + 4 + kDecWarps);
};

template <int TYPE, int NT, int PITCH>
struct __align__(1024) Smem {
  using S = Shape<TYPE, NT>;
  uint32_t tab[TYPE == T_IQ2_XXS ? kIq2Table : 256];      // first: its lookups count on the place
  uint8_t b[2][4][S::kBBytes];
  uint8_t bm[Fmt<TYPE>::mins ? 2 : 1][Fmt<TYPE>::mins ? S::kBBytes : 1024];      // sums of the token values, for the minima
  uint8_t ring[S::kSlots][BM * PITCH];
  float factor[4][Fmt<TYPE>::mins ? 2 : 1][BM];      // of a unit's rows, and those of the minima
  uint64_t raw[S::kSlots], freed[S::kSlots];      // a slot's blocks are there; have been read
  uint64_t full[2], done[2], folded[2];              // a unit's operands are there, its products are, its accumulator has been read
  uint64_t drained;
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
  uint32_t last[4];
  int prefix[kMaxGroups + 1];     // token tiles before each group
  int2 tiles[kMaxTiles];          // `Cursor::place`
};

// One stretch of work: blocks [b0, b1) of a tile of 128 weight rows and up to NT columns.
struct Item {
  int group, rt, split, b0, b1, row0, cnt, tile;
};

// A CTA's items in their order: parts of K within row tiles within token tiles, every gridDim.x-th of them.
template <int NT, int TERMS>
struct Cursor {
  int split, rt, tt;
  __device__ __forceinline__ explicit Cursor(const Params& p) {
    const int i = blockIdx.x / p.splits;
    split = blockIdx.x - i * p.splits;
    tt = i / p.row_tiles;
    rt = i - tt * p.row_tiles;
  }
  __device__ __forceinline__ void next(const Params& p) {
    split += p.step_split;
    rt += p.step_rt;
    tt += p.step_tt;
    if (split >= p.splits) {
      split -= p.splits;
      ++rt;
    }
    if (rt >= p.row_tiles) {
      rt -= p.row_tiles;
      ++tt;
    }
  }
  template <class Sm>
  __device__ __forceinline__ bool get(const Params& p, const Sm& sm, Item& w) const {
    if (tt >= sm.prefix[p.n_groups]) return false;
    w.split = split;
    w.rt = rt;
    w.tile = tt * p.row_tiles + rt;
    w.b0 = p.splits == 1 ? 0 : p.nblk * split / p.splits;
    w.b1 = p.splits == 1 ? p.nblk : p.nblk * (split + 1) / p.splits;
    const int2 t = tt < kMaxTiles ? sm.tiles[tt] : search(p, sm.prefix, tt);
    w.row0 = t.x;
    w.cnt = t.y & 255;
    w.group = t.y >> 8;
    return true;
  }
  static __device__ __forceinline__ int2 search(const Params& p, const int* prefix, int tt) {
    int lo = 0, hi = p.n_groups;      // prefix[lo] <= tt < prefix[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (prefix[mid] <= tt) lo = mid;
      else hi = mid;
    }
    return place(p, lo, tt - prefix[lo]);
  }
  // tile n of a group: first row; group * 256 + rows
  static __device__ __forceinline__ int2 place(const Params& p, int g, int n) {
    const int first = p.seg ? __ldg(p.seg + g) : 0, end = p.seg ? __ldg(p.seg + g + 1) : p.M, row0 = first + n * (NT / TERMS);
    return make_int2(row0, g * 256 + min(NT / TERMS, end - row0));
  }
};

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

// `__byte_perm` without its mask over the selector, whose nibbles are 0 to 7 here
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// A value that is kept in a register, not computed again at every use.
__device__ __forceinline__ void keep(uint32_t& v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ uint32_t mul2(uint32_t x, __half2 s, __half2 off) {
  const __half2 r = __hfma2(*reinterpret_cast<__half2*>(&x), s, off);
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <int OFF = 0>
__device__ __forceinline__ uint32_t ld_shared(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1 + %2];" : "=r"(v) : "r"(a), "n"(OFF) : "memory");
  return v;
}
__device__ __forceinline__ float half_of(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }
__device__ __forceinline__ uint4 ld_shared4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}

// `load`: what piece j of a lane's row needs, from the unit at `src`, whose first byte has the address a16 (mod 16) in memory.
// `half_piece`: sub-block h of the piece as 16 pairs in the order of the token rows. `factors`: those of the row's block.
template <int TYPE> struct Dec;
// A weight is one of three magnitudes with a sign: a nibble of 0..2 for the magnitude, plus 4 when it is negative. An entry's eight
// nibbles and a sign pattern's eight come from tables that hold every word once per lane (a random read is then one pass, where entries of
// 8 bytes read by 32 lanes took six on average), and the sum of the two selects bytes 128 +- magnitude by byte permutation. With 0x64
// above them these are halves 1024 + 128 +- magnitude; scale and bias are one fused multiply-add.
template <> struct Dec<T_IQ2_XXS> {
  // 66 bytes lie in five of the 16-byte pieces of memory, wherever they begin
  static constexpr int kPitch = 80, kRegs = 10;
  static constexpr uint32_t kAlign = 32768;      // of the tables: the place of an entry and of the lane are put together by bits
  // Rows in the ring: eight rows of 80 bytes are a multiple of all banks; rows of different alignment come to those places.
  __device__ static int place(int r) { return (r >> 2) | (r & 3) << 3; }
  __device__ static void load(uint32_t src, uint32_t a16, int j, uint32_t tab, uint32_t (&w)[kRegs]) {
    const uint32_t o = a16 + 2 + 16 * j, a = src + (o & ~3u), sel = (o & 2) ? 0x5432u : 0x3210u;
    uint32_t v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] = ld_shared(a + 4 * i);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t idx = prmt(v[2 * h], v[2 * h + 1], sel), aux = prmt(v[2 * h + 1], v[2 * h + 2], sel), aux2 = aux >> 14;
      w[8 + h] = aux;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const uint32_t si = g == 0 ? aux << 7 : g == 1 ? aux : g == 2 ? aux2 << 7 : aux2;
        w[4 * h + g] = ld_shared(tab + prmt(idx, 0, 0x4440 + g) * 128u) + ld_shared<32768>(tab | (si & 0x3f80u));
      }
    }
  }
  __device__ static void half_piece(const uint32_t (&w)[kRegs], int h, uint32_t (&x)[16]) {
    // the odd scale 2 s + 1 as a half, from 1024 + it
    const uint32_t lsw = 0x64016401u + (w[8 + h] >> 28) * 0x00020002u;
    const __half2 s2 = __hadd2(*reinterpret_cast<const __half2*>(&lsw), __float2half2_rn(-1024.f)), o2 = __hmul2(s2, __float2half2_rn(-1152.f));
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      constexpr uint32_t plus = 136u | 153u << 8 | 171u << 16, minus = 120u | 103u << 8 | 85u << 16;      // 128 +- 8, 25, 43
      const uint32_t c = w[4 * h + g], lo = prmt(plus, minus, c), hi = prmt(plus, minus, c >> 16);
      x[4 * g] = mul2(prmt(lo, 0x64646464u, 0x4140), s2, o2);
      x[4 * g + 1] = mul2(prmt(lo, 0x64646464u, 0x4342), s2, o2);
      x[4 * g + 2] = mul2(prmt(hi, 0x64646464u, 0x4140), s2, o2);
      x[4 * g + 3] = mul2(prmt(hi, 0x64646464u, 0x4342), s2, o2);
    }
  }
  __device__ static void factors(uint32_t src, uint32_t a16, float* f) { f[0] = 0.125f * half_of(ld_shared(src + (a16 & ~3u)) >> (8 * (a16 & 2))); }
  // Warp w of twelve writes 32 entries of the table.
  __device__ static void fill(uint32_t* tab, int w, int lane) {
    uint32_t c = 0;
    if (w < 8) {
      const uint64_t e = kIq2xxsGrid[32 * w + lane] >> 4;      // 8, 25, 43 -> 0, 1, 2
#pragma unroll
      for (int i = 0; i < 8; ++i) c |= (uint32_t)(e >> (8 * i) & 3u) << (4 * nibble(i));
    } else {
      const uint32_t n = 32 * (w - 8) + lane, sg = n | (__popc(n) & 1u) << 7;      // the eighth sign makes their number even
#pragma unroll
      for (int i = 0; i < 8; ++i) c |= (sg >> i & 1u) << (4 * nibble(i) + 2);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) tab[(32 * w + i) * 32 + lane] = __shfl_sync(0xffffffffu, c, i);
  }
  // of weight i of eight
  __host__ __device__ static constexpr int nibble(int i) { return (i & 4) | (i & 1) << 1 | (i & 2) >> 1; }
};

// scale (m = 0) or minimum (m = 1) of sub-block j from the twelve bytes of a K-quant's 6-bit pairs
__device__ __forceinline__ uint32_t k4_field(const uint32_t (&s)[3], int j, int m) {
  const int k = (j & 3) * 8;
  if (j < 4) return (s[m] >> k) & 63u;
  return ((s[2] >> (k + 4 * m)) & 15u) | (((s[m] >> (k + 6)) & 3u) << 4);
}

// K-quants: low and high nibbles of the 32 bytes of a piece are its two sub-blocks.
template <int TYPE> struct DecK {
  static constexpr int kPitch = Fmt<TYPE>::bytes, kRegs = TYPE == T_Q5_K ? 18 : 10;
  static constexpr uint32_t kAlign = 1024;
  __device__ static int place(int r) { return r; }
  // words 0 to 7: codes; then the scales of the sub-blocks; then Q5_K's high bits, those of the piece lowest in their bytes
  __device__ static void load(uint32_t src, uint32_t, int j, uint32_t, uint32_t (&w)[kRegs]) {
    const uint4 f = ld_shared4(src);
    const uint32_t s[3] = {f.y, f.z, f.w};
    w[8] = k4_field(s, 2 * j, 0);
    w[9] = k4_field(s, 2 * j + 1, 0);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint4 q = ld_shared4(src + (TYPE == T_Q5_K ? 48 : 16) + 32 * j + 16 * i);
      w[4 * i] = q.x;
      w[4 * i + 1] = q.y;
      w[4 * i + 2] = q.z;
      w[4 * i + 3] = q.w;
      if constexpr (TYPE == T_Q5_K) {
        const uint4 t = ld_shared4(src + 16 + 16 * i);
        w[10 + 4 * i] = t.x >> (2 * j);
        w[11 + 4 * i] = t.y >> (2 * j);
        w[12 + 4 * i] = t.z >> (2 * j);
        w[13 + 4 * i] = t.w >> (2 * j);
      }
    }
  }
  __device__ static void half_piece(const uint32_t (&w)[kRegs], int h, uint32_t (&x)[16]) {
    const int c = (int)w[8 + h];
    const __half2 s2 = __half2half2(__int2half_rn(c)), o2 = __half2half2(__int2half_rn((h ? -64 : -1024) * c));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = w[i], q8 = q >> 8;
      uint32_t a0, a1;
      if (h == 0) {      // 1024 + code
        a0 = (q & 0x000f000fu) | 0x64006400u;
        a1 = (q8 & 0x000f000fu) | 0x64006400u;
      } else {           // 64 + code
        a0 = (q & 0x00f000f0u) | 0x54005400u;
        a1 = (q8 & 0x00f000f0u) | 0x54005400u;
      }
      if constexpr (TYPE == T_Q5_K) {
        const uint32_t t = w[10 + i], t8 = t >> 8;      // bit 0: low sub-block, bit 1: high
        a0 |= h ? (t << 7) & 0x01000100u : (t << 4) & 0x00100010u;
        a1 |= h ? (t8 << 7) & 0x01000100u : (t8 << 4) & 0x00100010u;
      }
      x[2 * i] = mul2(a0, s2, o2);
      x[2 * i + 1] = mul2(a1, s2, o2);
    }
  }
  __device__ static void factors(uint32_t src, uint32_t, float* f) {
    const uint32_t v = ld_shared(src);
    f[0] = half_of(v);
    f[BM] = -half_of(v >> 16);
  }
  // the codes of the eight minima, for the sums' first and second terms
  __device__ static void minima(uint32_t src, uint32_t (&x)[8]) {
    const uint4 f = ld_shared4(src);
    const uint32_t s[3] = {f.y, f.z, f.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 v = __halves2half2(__uint2half_rn(k4_field(s, 2 * i, 1)), __uint2half_rn(k4_field(s, 2 * i + 1, 1)));
      x[i] = x[i + 4] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
};
template <> struct Dec<T_Q4_K> : DecK<T_Q4_K> {};
template <> struct Dec<T_Q5_K> : DecK<T_Q5_K> {};

// E4M3 codes are fp16 numbers already; a unit is two tiles of 128 bytes a row in the 128-byte swizzle (bank conflicts).
template <> struct Dec<T_E4M3> {
  static constexpr int kPitch = 256, kRegs = 16;
  static constexpr uint32_t kAlign = 1024;
  __device__ static int place(int r) { return r; }
  __device__ static void load(uint32_t src, uint32_t, int j, uint32_t, uint32_t (&w)[kRegs]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 v = ld_shared4((src + (j >> 1) * (BM * 128)) + ((64 * (j & 1) + 16 * i) ^ (src >> 3 & 0x70)));
      w[4 * i] = v.x;
      w[4 * i + 1] = v.y;
      w[4 * i + 2] = v.z;
      w[4 * i + 3] = v.w;
    }
  }
  __device__ static void half_piece(const uint32_t (&w)[kRegs], int h, uint32_t (&x)[16]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t v = w[8 * h + i];
      const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v & 0xffffu), __NV_E4M3);
      const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v >> 16), __NV_E4M3);
      x[2 * i] = (uint32_t)lo.x | (uint32_t)lo.y << 16;
      x[2 * i + 1] = (uint32_t)hi.x | (uint32_t)hi.y << 16;
    }
  }
};

// By the fold warps of a quarter of the rows, behind their stores of a part: whether the other parts of these rows are there. A byte
// of the tile's counter per quarter, so that quarters do not wait for one another.
template <int WARPS>
__device__ __forceinline__ bool count_part(const Params& p, const Item& w, uint32_t* last) {
  const int q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  auto sync = [&]() {
    if constexpr (WARPS == 8) asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
    else __syncwarp();
  };
  sync();
  if (threadIdx.x < 128 && lane == 0) {
    uint32_t n;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(n) : "l"(p.counters + w.tile), "r"(1u << (8 * q)) : "memory");
    last[q] = ((n >> (8 * q)) & 255u) == (uint32_t)p.splits - 1u;
    if (last[q]) atomicSub(p.counters + w.tile, (uint32_t)p.splits << (8 * q));
  }
  sync();
  return *(volatile uint32_t*)&last[q];
}

// The rest of a fold warp's items, from `cur` on, after a wait that ran out: NaN in their places, so that the result cannot be taken
// for one, and every part counted, so that the counters are back at zero when the launch is over. Kept out of the loop that it ends.
template <int NT, int TERMS, int WARPS, class Sm>
__device__ __noinline__ void give_up(const Params& p, Sm& sm, Cursor<NT, TERMS> cur, int c0) {
  const int tid = threadIdx.x, lr = ((tid >> 5) & 3) * 32 + (tid & 31), cols = WARPS == 8 ? NT / 2 : NT;
  const float nan = __uint_as_float(0x7fffffffu);
  Item w;
  for (; cur.get(p, sm, w); cur.next(p)) {
    if (p.splits > 1) {
      float* part = p.ws + ((size_t)w.tile * p.splits + w.split) * NT * BM + lr;
      for (int c = c0; c < c0 + cols; ++c) __stcg(part + (size_t)c * BM, nan);
      if (!count_part<WARPS>(p, w, sm.last)) continue;
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

// The copies that this thread has begun arrive on `bar` when they are there.
__device__ __forceinline__ void copies_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)), "l"(map),
               "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}

// Before `pdl_wait` the kernel reads the weights and the route segments: its predecessor in the stream is the staging of its rows (or
// another product of them), which lets it begin only when everything before itself is complete. What is left of that launch, a few us, counts in the limits
// of the waits.
template <int TYPE, int NT, int TERMS>
__global__ void __launch_bounds__(Shape<TYPE, NT>::kThreads, 1)
quant_umma_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ Params p) {
  using S = Shape<TYPE, NT>;
  constexpr int BB = Fmt<TYPE>::bytes;
  constexpr bool MINS = Fmt<TYPE>::mins;
  constexpr int kPieces = Fmt<TYPE>::k / 64, kUnit = 4 / kPieces;      // pieces of a block, blocks of a unit
  // One CTA can have several parts of K where a decode step uses it (16 columns; wider tiles have no registers for it).
  constexpr bool kParts = TYPE != T_E4M3 && NT == 16;
  // Tensor memory: accumulators of two units, that of the minima, the sum of the parts, the codes of the minima of two units, the weights of two units.
  constexpr uint32_t kAccCols = kUnit * NT, kMinCol = 2 * NT, kSumCol = 3 * NT, kACodes = 240, kACol = 256, kTmemCols = 512;
  static_assert(2 * kAccCols <= kACol && (TYPE == T_E4M3 || 3 * NT + (kParts ? NT : 0) <= kACodes), "tensor memory");
  extern __shared__ uint8_t smem_raw[];
  using D = Dec<TYPE>;
  using Sm = Smem<TYPE, NT, D::kPitch>;
  // aligned in the shared window, whose addresses the lookups are made of
  Sm& sm = *reinterpret_cast<Sm*>(smem_raw + (-smem_u32(smem_raw) & (D::kAlign - 1)));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  using Cur = Cursor<NT, TERMS>;

  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.full[b], S::kDecWarps + 1);
      mbar_init(&sm.done[b], 1);
      mbar_init(&sm.folded[b], S::kFoldWarps);
    }
    for (int k = 0; k < S::kSlots; ++k) {
      mbar_init(&sm.raw[k], TYPE == T_IQ2_XXS ? 64 : 1);
      mbar_init(&sm.freed[k], 1);
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
    if (warp >= 4 && warp < 16) D::fill(sm.tab, warp - 4, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;
  for (int g = warp; g < p.n_groups; g += S::kThreads / 32) {
    const int first = sm.prefix[g], n = min(sm.prefix[g + 1], kMaxTiles) - first;
    for (int k = lane; k < n; k += 32) sm.tiles[first + k] = Cur::place(p, g, k);
  }
  __syncthreads();

  if (warp < S::kFoldWarps) {
    // ---------------- fold and epilogue ----------------
    pk::pdl_wait();
    pk::pdl_trigger();
    const int q = warp & 3, c0 = (warp >> 2) * S::kFoldCols, lr = q * 32 + lane;
    uint32_t unit = 0;
    Item w;
    bool ok = true;
    // an earlier product of the step gave up: this one does as if its first wait had
    const bool dead = p.status != nullptr && __any_sync(0xffffffffu, *(const volatile uint32_t*)p.status);
    if (dead) sm.abort_flag = 1u;
    for (Cur cur(p); ok && cur.get(p, sm, w); cur.next(p)) {
      float acc[S::kFoldCols];
#pragma unroll
      for (int c = 0; c < S::kFoldCols; ++c) acc[c] = 0.f;
      const float* ws = nullptr;
      if constexpr (TYPE == T_E4M3) {
        const int half = p.rows >> 1;
        const int r = (p.epi & 1) ? min(w.rt * 64 + (lr >> 1), half - 1) + (lr & 1) * half : w.rt * BM;
        ws = p.w_scale + (size_t)(r >> 7) * p.w_ld;
      }
      [[maybe_unused]] int part = 0, part_end = kParts && p.splits == 1 && p.parts > 1 ? p.nblk / p.parts : -1;
      for (int b = w.b0; b < w.b1; b += kUnit, ++unit) {
        const int buf = unit & 1;
        if (dead || !mbar_wait_uniform(&sm.done[buf], (unit >> 1) & 1, &sm.abort_flag, p.status, 31)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll 1
        for (int k = 0; k < kUnit; ++k) {
          if (kUnit > 1 && b + k >= w.b1) break;
          const float f = TYPE == T_E4M3 ? __ldg(ws + b + k) : sm.factor[unit & 3][0][lr];
          const uint32_t t = tmem_base + c0 + ((uint32_t)(q * 32) << 16);
#pragma unroll
          for (int c = 0; c < S::kFoldCols; c += 16) {
            uint32_t r[16];
            tmem_ld_32x16(t + buf * kAccCols + k * NT + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(f, __uint_as_float(r[j]), acc[c + j]);
            if constexpr (MINS) {
              const float fm = sm.factor[unit & 3][1][lr];
              tmem_ld_32x16(t + kMinCol + c, r);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(fm, __uint_as_float(r[j]), acc[c + j]);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.folded[buf]);
        if constexpr (kParts)
          if (b + 1 == part_end) {
            const uint32_t ts = tmem_base + kSumCol + ((uint32_t)(q * 32) << 16);
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
        give_up<NT, TERMS, S::kFoldWarps>(p, sm, cur, c0);
        break;
      }
      if (p.splits > 1) {
        float* part = p.ws + ((size_t)w.tile * p.splits + w.split) * NT * BM + lr;
#pragma unroll
        for (int c = 0; c < S::kFoldCols; ++c) __stcg(part + (size_t)(c0 + c) * BM, acc[c]);
        if (!count_part<S::kFoldWarps>(p, w, sm.last)) continue;
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
        if (m0 + m < w.cnt) v[m] *= p.row_scale[w.row0 + m0 + m];
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
    const uint64_t db0 = smem_desc_k_sw128(smem_u32(sm.b[0][0])), dm0 = smem_desc_k_sw128(smem_u32(sm.bm[0]));
    const bool leader = elect_one();
    uint32_t unit = 0, slot = 0;
    Item w;
    bool ok = true;
    for (Cur cur(p); ok && cur.get(p, sm, w); cur.next(p)) {
      for (int b = w.b0; b < w.b1; b += kUnit, ++unit) {
        const uint32_t buf = unit & 1, ph = (unit >> 1) & 1;
        // the one accumulator of the minima: the fold is through with the unit before, too
        ok = mbar_wait_uniform(&sm.folded[buf], ph ^ 1, &sm.abort_flag, p.status, 32) && mbar_wait_uniform(&sm.full[buf], ph, &sm.abort_flag, p.status, 33) &&
             (!MINS || unit == 0 || mbar_wait_uniform(&sm.folded[buf ^ 1], ((unit - 1) >> 1) & 1, &sm.abort_flag, p.status, 34));
        if (!ok) break;
        if (TYPE == T_IQ2_XXS && leader) mbar_arrive(&sm.freed[slot]);      // full: all decode warps have read theirs
        slot = slot + 1 == S::kSlots ? 0 : slot + 1;
        tc_fence_after();
        const uint32_t acc = tmem_base + buf * kAccCols, ta = tmem_base + kACol + buf * 128;
        const uint64_t db = db0 + buf * (4 * S::kBBytes >> 4);
        const int pieces = kUnit == 1 ? 4 : min(4, (w.b1 - b) * kPieces);      // the last unit of an item can be one E4M3 block
        if (leader) {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (kUnit == 1 || k / 4 < pieces)
              umma_f16_ts(acc + (k / (4 * kPieces)) * NT, ta + k * 8, db + (k / 4) * (S::kBBytes >> 4) + (k % 4) * 2, idesc, k % (4 * kPieces) > 0 ? 1u : 0u);
          if constexpr (MINS) umma_f16_ts(tmem_base + kMinCol, tmem_base + kACodes + buf * 8, dm0 + buf * (S::kBBytes >> 4), idesc, 0u);
          umma_commit(&sm.done[buf]);
        }
        __syncwarp();
      }
    }
    if (!ok) {
      // gave up: the products in flight end before their tensor memory is freed
      if (leader) umma_commit(&sm.drained);
      __syncwarp();
      for (uint32_t n = 0; n < kDrainPolls && !mbar_try_wait(&sm.drained, 0); ++n) {}
    }
  } else if (warp == S::kFoldWarps + 1) {
    // ---------------- token tiles, raw blocks whose rows are whole 16 bytes ----------------
    if (lane == 0) {
      tma_prefetch_desc(&tmap);
      constexpr bool RAW = TYPE != T_IQ2_XXS;
      constexpr uint32_t kBlockBytes = BM * BB;
      // Raw blocks run kSlots units ahead, over the ends of the CTA's items.
      Cur ahead(p);
      Item c;
      c.b0 = c.b1 = 0;
      uint32_t fill = 0, copied = 0;
      auto copy_next = [&]() {
        if (c.b0 >= c.b1) {
          if (!ahead.get(p, sm, c)) return;
          ahead.next(p);
        }
        const int blocks = min(kUnit, c.b1 - c.b0), row = c.rt * ((p.epi & 1) ? 64 : BM);
        mbar_arrive_expect_tx(&sm.raw[fill], blocks * kBlockBytes);
        for (int k = 0; k < blocks; ++k) tma_load_4d(sm.ring[fill] + k * kBlockBytes, &wmap, &sm.raw[fill], (c.b0 + k) * BB, 0, row, c.group);
        c.b0 += kUnit;
        ++copied;
        fill = fill + 1 == S::kSlots ? 0 : fill + 1;
      };
      if constexpr (RAW)
        for (int k = 0; k < S::kSlots; ++k) copy_next();
      pk::pdl_wait();      // the staged rows
      uint32_t unit = 0;
      Item w;
      bool ok = true;
      for (Cur cur(p); ok && cur.get(p, sm, w); cur.next(p))
        for (int b = w.b0; b < w.b1; b += kUnit, ++unit) {
          const uint32_t buf = unit & 1;
          if (!mbar_wait(&sm.done[buf], ((unit >> 1) & 1) ^ 1, &sm.abort_flag, p.status, 35)) {
            ok = false;
            break;
          }
          const int pieces = kUnit == 1 ? 4 : min(4, (w.b1 - b) * kPieces), x = b * Fmt<TYPE>::cols;
          mbar_arrive_expect_tx(&sm.full[buf], (pieces + (MINS ? 1 : 0)) * NT * 128);
          for (int j = 0; j < pieces; ++j) tma_load_2d(sm.b[buf][j], &tmap, &sm.full[buf], x + 64 * j, w.row0 * TERMS);
          if constexpr (MINS) tma_load_2d(sm.bm[buf], &tmap, &sm.full[buf], x + 256, w.row0 * TERMS);
          if (RAW && unit >= 2) copy_next();      // into the slot of the unit that has been multiplied
        }
      if (sm.abort_flag) {
        // gave up: copies in flight land before the CTA exits
        for (uint32_t u = unit > 2 ? unit - 2 : 0; u < unit; ++u)
          for (uint32_t n = 0; n < kDrainPolls; ++n)
            if (mbar_try_wait(&sm.full[u & 1], (u >> 1) & 1)) break;
        if constexpr (RAW)
          for (uint32_t u = copied > S::kSlots ? copied - S::kSlots : 0; u < copied; ++u)
            for (uint32_t n = 0; n < kDrainPolls; ++n)
              if (mbar_try_wait(&sm.raw[u % S::kSlots], (u / S::kSlots) & 1)) break;
      }
    }
  } else if (warp < S::kFoldWarps + 4) {
    // ---------------- raw blocks of 66 bytes: two warps, 64 rows each ----------------
    // Five 16-byte pieces of memory hold a block, wherever it begins (those at its ends hold bytes of its neighbours). Bulk copies of 80
    // bytes take 35 cycles each, several times the decode; as two warps' work `cp.async` costs the decode warps nothing.
    if constexpr (TYPE == T_IQ2_XXS) {
      constexpr int kCopies = 10;
      const int r0 = (warp - S::kFoldWarps - 2) * 64;
      uint32_t to[kCopies], off[kCopies];
#pragma unroll
      for (int k = 0; k < kCopies; ++k) {
        const int n = lane + 32 * k, r = r0 + n / 5;
        to[k] = smem_u32(sm.ring[0]) + ((r & ~31) + D::place(r & 31)) * D::kPitch + n % 5 * 16;
        keep(to[k]);
      }
      const uint8_t* pos = p.W;
      int left = 0;      // blocks of the cursor's item
      uint32_t fill = 0, turn = 0;
      Item c;
      Cur ahead(p);
      while (true) {
        if (left == 0) {
          if (!ahead.get(p, sm, c)) break;
          ahead.next(p);
          left = c.b1 - c.b0;
          pos = group_base(p, c) + c.b0 * BB;
#pragma unroll
          for (int k = 0; k < kCopies; ++k) off[k] = tile_row(p, c, r0 + (lane + 32 * k) / 5) + (lane + 32 * k) % 5 * 16;
        }
        if (!mbar_wait_uniform(&sm.freed[fill], turn ^ 1, &sm.abort_flag, p.status, 38)) break;
        const uint32_t at = fill * (BM * D::kPitch);
#pragma unroll
        for (int k = 0; k < kCopies; ++k)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to[k] + at), "l"((uintptr_t)(pos + off[k]) & ~(uintptr_t)15) : "memory");
        copies_arrive(&sm.raw[fill]);
        --left;
        pos += BB;
        if (++fill == S::kSlots) {
          fill = 0;
          turn ^= 1u;
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    // ---------------- decode ----------------
    // A lane has a row of its warp's quarter, the only rows whose tensor memory the warp can write, and piece j of every unit.
    const int q = warp & 3, j = (warp - S::kFoldWarps - 4) >> 2, lr = q * 32 + lane;
    uint32_t tab = smem_u32(sm.tab) + lane * 4, ta0 = tmem_base + kACol + ((uint32_t)(q * 32) << 16) + j * 32;
    const uint32_t row = smem_u32(sm.ring[0]) + (q * 32 + D::place(lane)) * (TYPE == T_E4M3 ? 128 : D::kPitch);
    uint32_t unit = 0, slot = 0, turn = 0;
    keep(tab);
    keep(ta0);
    Item w;
    bool ok = true;
    for (Cur cur(p); ok && cur.get(p, sm, w); cur.next(p)) {
      uint32_t at = (uint32_t)(uintptr_t)group_base(p, w) + tile_row(p, w, lr) + w.b0 * BB;      // address of the unit, its last bits
      for (int b = w.b0; b < w.b1; b += kUnit, ++unit, at += kUnit * BB) {
        if (!mbar_wait_uniform(&sm.raw[slot], turn, &sm.abort_flag, p.status, 37)) {
          ok = false;
          break;
        }
        const uint32_t src = row + slot * (BM * D::kPitch), a16 = at & 15u, buf = unit & 1, ta = ta0 + buf * 128;
        if (++slot == S::kSlots) {
          slot = 0;
          turn ^= 1u;
        }
        uint32_t raw[D::kRegs], x[16];
        D::load(src, a16, j, tab, raw);
        if (!mbar_wait_uniform(&sm.done[buf], ((unit >> 1) & 1) ^ 1, &sm.abort_flag, p.status, 36)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // four units of factors: the fold has read those of the unit four back when the one two back has been multiplied
        if constexpr (TYPE != T_E4M3)
          if (j == 0) D::factors(src, a16, &sm.factor[unit & 3][0][lr]);
        D::half_piece(raw, 0, x);
        tmem_st_32x16(ta, x);
        D::half_piece(raw, 1, x);
        tmem_st_32x16(ta + 16, x);
        if constexpr (MINS)
          if (j == 3) {
            uint32_t m[8];
            D::minima(src, m);
            tmem_st_32x8(tmem_base + kACodes + buf * 8 + ((uint32_t)(q * 32) << 16), m);
          }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.full[buf]);
      }
    }
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
  pk::pdl_wait();
  pk::pdl_trigger();
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
  CUtensorMap map, wmap{};
  const cuuint64_t pitch = (cuuint64_t)p.nblk * Fmt<TYPE>::cols;
  const cuuint64_t gdim[2] = {pitch, (cuuint64_t)total_rows * TERMS}, gstride[1] = {pitch * 2};
  const cuuint32_t box[2] = {64, NT}, estr[4] = {1, 1, 1, 1};
  if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(staged), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return PK_ERR_CUDA;
  if constexpr (TYPE != T_IQ2_XXS) {
    // bytes of a row, gate and up of a pair (or one), rows, groups; every stride is a multiple of a block's bytes, which are whole 16
    const cuuint64_t two = (p.epi & 1) ? 2 : 1, rows = p.rows / two, rb = (cuuint64_t)p.rb;
    const cuuint64_t wdim[4] = {rb, two, rows, (cuuint64_t)p.n_groups}, wstride[3] = {rows * rb, rb, rb * p.rows};
    const cuuint32_t wbox[4] = {(cuuint32_t)Fmt<TYPE>::bytes, (cuuint32_t)two, (cuuint32_t)(BM / two), 1};
    if (encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<uint8_t*>(p.W), wdim, wstride, wbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               TYPE == T_E4M3 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return PK_ERR_CUDA;
  }
  constexpr size_t smem = sizeof(Smem<TYPE, NT, Dec<TYPE>::kPitch>) + Dec<TYPE>::kAlign;
  static_assert(smem <= 227 * 1024, "shared memory");
  static PkDeviceOnce once;
  if (PkDeviceOnceGuard once_guard{once}; once_guard.needed()) {
    if (cudaFuncSetAttribute(quant_umma_kernel<TYPE, NT, TERMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      pk_set_last_cuda_error((int)cudaGetLastError());
      return PK_ERR_CUDA;
    }
    once_guard.done();
  }
  PK_LAUNCH_PDL((quant_umma_kernel<TYPE, NT, TERMS>), dim3(sms), dim3(Shape<TYPE, NT>::kThreads), smem, stream, map, wmap, p);
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
  PK_LAUNCH_PDL(quant_stage_rows_kernel, dim3(rows), dim3(threads), smem, stream, p);
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
  if (splits > 255) parts = splits = 255;      // a byte counts them
  const int sms = sm_count > 0 ? sm_count : 148;
  const int row_tiles = (epi & 1) ? (N / 2 + 63) / 64 : (N + BM - 1) / BM;
  const Params p{(const uint8_t*)W, (long long)nblk * type_bytes(type), nblk, N, n_groups, seg, rows, epi, limit, out, ldo, (const pk::bf16*)resid, row_scale, w_scale, w_ld,
                 parts, splits, ws, counters, status, row_tiles, sms % splits, sms / splits % row_tiles, sms / splits / row_tiles};
  if (type == T_IQ2_XXS) return launch_shape<T_IQ2_XXS>(columns, terms, staged, rows, p, sms, stream);
  if (type == T_Q4_K) return launch_shape<T_Q4_K>(columns, terms, staged, rows, p, sms, stream);
  if (type == T_Q5_K) return launch_shape<T_Q5_K>(columns, terms, staged, rows, p, sms, stream);
  if (columns == 32) return launch<T_E4M3, 32, 1>(staged, rows, p, sms, stream);
  return launch<T_E4M3, 64, 1>(staged, rows, p, sms, stream);
}
