// Work space of the stream-K schedules (gemm_bf16.cu, gemm_fp8.cu): partial tiles of a launch's CTAs and the flags that publish them.
#pragma once

#include <cstdlib>
#include <mutex>

#include "pk_common.cuh"

namespace pk {

struct StreamK {
  float* ws = nullptr;          // [ctas][128 * 256]
  uint32_t* flags = nullptr;    // [ctas]: number of the launch whose partial is in ws
  uint32_t seq = 0;             // this launch's
};

// The schedule is taken where `streamk_pays` says so; POCKET_GEMM_NO_STREAMK or POCKET_GEMM_STREAMK=0 turn it off, POCKET_GEMM_STREAMK=1 takes it
// wherever whole tiles would leave SMs idle and a group of CTAs gets some blocks.
enum class StreamKMode { never, cost, forced };
inline StreamKMode streamk_mode() {
  if (getenv("POCKET_GEMM_NO_STREAMK") != nullptr) return StreamKMode::never;
  const char* v = getenv("POCKET_GEMM_STREAMK");
  return v == nullptr ? StreamKMode::cost : v[0] == '1' ? StreamKMode::forced : StreamKMode::never;
}

// Allocations that another thread's capture does not mind.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Whether sharing pays: what whole tiles take against what the groups of CTAs take, in blocks of K, against the exchange of the parts. The
// constants are fits to 174 (FP8) and 97 (bf16) shapes of 65 to 3000 rows, each timed both ways; with them the slower way is taken in one of them
// by more than 5 % (with whole tiles throughout 9 and 11 % are lost in the mean, with sharing throughout 6 %). us, whole tiles / shared: FP8,
// two terms, 512 rows, K x 5120, K = 1536 17 / 24, 2176 20 / 26, 4096 45 / 43, 17408 108 / 88; 2048 rows of 12288 x 5120 208 / 231; 128 rows, K = 17408,
// 123 / 59; bf16, 300 rows of 10304 x 4096 36 / 39, 1900 of 1088 x 1024 14 / 19, 168 of 10304 x 4096 45 / 43.
struct StreamKCost {
  int least;                      // blocks of a group
  double fixed, part, share;      // of the exchange, for each part of a tile, for each block of a group
};
inline bool streamk_pays(int tiles_m, int tiles_n, int num_kb, int sms, const StreamKCost& c) {
  const StreamKMode mode = streamk_mode();
  const int tiles = tiles_m * tiles_n, rounds = (tiles + sms - 1) / sms, groups = tiles_m <= sms ? sms / tiles_m : 0;
  if (mode == StreamKMode::never || groups < 2 || tiles >= 0.88 * rounds * sms || (long long)tiles_n * num_kb < (long long)groups * c.least) return false;
  if (mode == StreamKMode::forced) return true;
  const double shared = (double)tiles_n * num_kb / groups, parts = groups > tiles_n ? (double)groups / tiles_n : 1.;
  return (double)rounds * num_kb - shared > c.fixed + c.part * parts + c.share * shared;
}

// Work spaces by stream, since launches on several streams can run at the same time: at most `kStreamKStreams` per device (19 MB each with
// 148 SMs), one for each of the first streams that ask. The streams after them work whole tiles, and so does every stream under capture (a
// replay would find the flags of the one before it): no launch waits for another stream. An owner of a stream can have its work space
// allocated ahead, and frees it when the stream has ended; the others live as long as the process, like the streams of torch's pool that have them.
constexpr int kStreamKStreams = 8;
struct StreamKPool {
  struct Entry {
    unsigned long long id = 0;
    StreamK b;      // b.ws null: no one's
    int ctas = 0;
  };
  std::mutex mu;
  Entry entries[64][kStreamKStreams];

  // The stream's entry, a new one where it has none and `make`; null without one. With `mu` held.
  Entry* of(cudaStream_t stream, int ctas, bool make) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    int dev = 0;
    unsigned long long id = 0;
    // (under capture nothing else is asked of the stream: its number would end the capture)
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || (capture == cudaStreamCaptureStatusNone && (cudaGetDevice(&dev) != cudaSuccess || cudaStreamGetId(stream, &id) != cudaSuccess))) {
      cudaGetLastError();
      return nullptr;
    }
    if (capture != cudaStreamCaptureStatusNone || dev < 0 || dev >= 64) return nullptr;
    Entry* empty = nullptr;
    for (Entry& x : entries[dev]) {
      if (x.b.ws != nullptr && x.id == id) return &x;
      if (x.b.ws == nullptr) empty = &x;
    }
    if (!make || empty == nullptr) return nullptr;
    RelaxedCapture relaxed;
    const int n = ctas > 148 ? ctas : 148;
    StreamK b;
    // cleared on the stream itself: its launches come behind, whatever the others do
    const bool ok = cudaMalloc(&b.ws, (size_t)n * 128 * 256 * sizeof(float)) == cudaSuccess && cudaMalloc(&b.flags, n * sizeof(uint32_t)) == cudaSuccess &&
                    cudaMemsetAsync(b.flags, 0, n * sizeof(uint32_t), stream) == cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      cudaFree(b.ws);
      cudaFree(b.flags);
      return nullptr;
    }
    empty->id = id;
    empty->b = b;
    empty->ctas = n;
    return empty;
  }
  void free(Entry& e) {
    RelaxedCapture relaxed;
    cudaFree(e.b.ws);
    cudaFree(e.b.flags);
    e = Entry();
  }
};
inline StreamKPool& streamk_pool() {
  static StreamKPool pool;
  return pool;
}

// The work space of a launch of `ctas` CTAs on `stream`; false: whole tiles.
inline bool streamk_take(int ctas, cudaStream_t stream, StreamK& out) {
  StreamKPool& pool = streamk_pool();
  std::lock_guard<std::mutex> lock(pool.mu);
  StreamKPool::Entry* e = pool.of(stream, ctas, true);
  if (e == nullptr || e->ctas < ctas) return false;
  ++e->b.seq;
  out = e->b;
  return true;
}

}  // namespace pk
