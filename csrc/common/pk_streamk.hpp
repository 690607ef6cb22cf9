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

// Work spaces by stream, since launches on several streams can run at the same time: at most `kStreamKStreams` per device (19 MB each with
// 148 SMs). An owner of a stream can reserve one and gives it back when the stream has ended; otherwise a stream's first launch
// allocates one or, when there are no more, takes that of a stream which has not been used for some time, after waiting for the device.
constexpr int kStreamKStreams = 8, kStreamKIdle = 64;
constexpr unsigned long long kStreamKFree = ~0ull;
struct StreamKPool {
  struct Entry {
    unsigned long long id = kStreamKFree, last = 0;
    StreamK b;
    int ctas = 0;
  };
  std::mutex mu;
  Entry entries[64][kStreamKStreams];
  unsigned long long launches = 0;

  // The stream's entry, a new one where it has none; null without one, and under capture (a replay would find the flags of the one
  // before it). With `mu` held.
  Entry* of(cudaStream_t stream, int ctas, bool make) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    int dev = 0;
    unsigned long long id = 0;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess || cudaStreamGetId(stream, &id) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (capture != cudaStreamCaptureStatusNone || dev < 0 || dev >= 64) return nullptr;
    Entry *unowned = nullptr, *empty = nullptr, *oldest = entries[dev];
    for (Entry& x : entries[dev]) {
      if (x.b.ws != nullptr && x.id == id) return &x;
      if (x.b.ws == nullptr) empty = &x;
      else if (x.id == kStreamKFree) unowned = &x;
      if (x.last < oldest->last) oldest = &x;
    }
    if (!make) return nullptr;
    Entry* e = unowned != nullptr ? unowned : empty;
    if (e == nullptr && oldest->last + kStreamKIdle > launches) return nullptr;
    if (unowned == nullptr) {
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // another thread may be capturing
      cudaThreadExchangeStreamCaptureMode(&mode);
      bool ok = true;
      if (e == nullptr) {
        e = oldest;
        ok = cudaDeviceSynchronize() == cudaSuccess;
      } else {
        const int n = ctas > 148 ? ctas : 148;
        StreamK b;
        ok = cudaMalloc(&b.ws, (size_t)n * 128 * 256 * sizeof(float)) == cudaSuccess && cudaMalloc(&b.flags, n * sizeof(uint32_t)) == cudaSuccess &&
             cudaMemset(b.flags, 0, n * sizeof(uint32_t)) == cudaSuccess;
        if (ok) {
          e->b = b;
          e->ctas = n;
        } else {
          cudaFree(b.ws);
          cudaFree(b.flags);
        }
      }
      if (!ok) cudaGetLastError();
      cudaThreadExchangeStreamCaptureMode(&mode);
      if (!ok) return nullptr;
    }
    e->id = id;
    e->last = launches;
    return e;
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
  ++pool.launches;
  StreamKPool::Entry* e = pool.of(stream, ctas, true);
  if (e == nullptr || e->ctas < ctas) return false;
  e->last = pool.launches;
  ++e->b.seq;
  out = e->b;
  return true;
}

}  // namespace pk
