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

// The schedule is the default wherever whole tiles would leave SMs idle; POCKET_GEMM_NO_STREAMK or POCKET_GEMM_STREAMK=0 turn it off.
inline bool streamk_allowed() {
  if (getenv("POCKET_GEMM_NO_STREAMK") != nullptr) return false;
  const char* v = getenv("POCKET_GEMM_STREAMK");
  return v == nullptr || v[0] != '0';
}

// Allocations that another thread's capture does not mind.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

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
