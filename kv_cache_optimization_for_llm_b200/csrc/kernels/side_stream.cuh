// A stream beside the caller's, for launches that touch nothing of the caller's next ones.  kvb_side_fork orders the side stream behind
// everything that the caller's stream holds so far, kvb_side_join orders what the caller's stream gets next behind the side stream.
// Ordinary events, so every kernel on either stream finds what it reads complete before it starts, and a captured graph gets two branches.
//
// One side stream per (device, caller's stream), made at its first use and kept, 32 at most: beyond that the one that was used longest
// ago is given back, unless somebody is between a fork and a join on it or it belongs to a capture.  Threads may share a stream: a fork's
// record and wait are one step, and so are a join's.
#pragma once

#include "common.cuh"

#include <mutex>
#include <vector>

namespace side {

struct Side {
  int device;
  cudaStream_t main, beside;
  cudaEvent_t fork, join;
  int open;                      // forks without their join
  unsigned long long used;
};

inline std::mutex& guard() { static std::mutex m; return m; }
inline std::vector<Side>& all() { static std::vector<Side> v; return v; }
constexpr size_t kMost = 32;

// Streams and events may be made while some stream of the process is being captured.
struct Relaxed {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

inline void give_back(Side& s) {
  cudaStreamDestroy(s.beside);   // (what it still holds runs to its end)
  cudaEventDestroy(s.fork);
  cudaEventDestroy(s.join);
}

// The caller's side stream; null: none could be made.  The guard is held.
inline Side* find(cudaStream_t main, bool make, cudaError_t& e) {
  static unsigned long long clock = 0;
  int device = 0;
  if ((e = cudaGetDevice(&device)) != cudaSuccess) return nullptr;
  std::vector<Side>& v = all();
  for (Side& s : v)
    if (s.device == device && s.main == main) { s.used = ++clock; return &s; }
  if (!make) { e = cudaErrorInvalidValue; return nullptr; }
  Relaxed relaxed;
  if (v.size() >= kMost) {
    size_t oldest = v.size();
    for (size_t i = 0; i < v.size(); ++i) {
      cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
      if (v[i].open == 0 && (oldest == v.size() || v[i].used < v[oldest].used) &&
          cudaStreamIsCapturing(v[i].beside, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone)
        oldest = i;
    }
    if (oldest < v.size()) {
      give_back(v[oldest]);
      v.erase(v.begin() + (long)oldest);
    }
  }
  Side s = {device, main, nullptr, nullptr, nullptr, 0, ++clock};
  if ((e = cudaStreamCreateWithFlags(&s.beside, cudaStreamNonBlocking)) != cudaSuccess) return nullptr;
  if ((e = cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming)) != cudaSuccess) { cudaStreamDestroy(s.beside); return nullptr; }
  if ((e = cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming)) != cudaSuccess) {
    cudaEventDestroy(s.fork);
    cudaStreamDestroy(s.beside);
    return nullptr;
  }
  v.push_back(s);
  return &v.back();
}

}  // namespace side

// *beside: the stream for what shall run beside the caller's next launches.  Every fork that returned 0 has its join.
KVB_EXPORT int kvb_side_fork(cudaStream_t stream, cudaStream_t* beside) {
  std::lock_guard<std::mutex> hold(side::guard());
  cudaError_t e = cudaSuccess;
  side::Side* s = side::find(stream, true, e);
  if (s == nullptr) return (int)e;
  if ((e = cudaEventRecord(s->fork, stream)) != cudaSuccess || (e = cudaStreamWaitEvent(s->beside, s->fork, 0)) != cudaSuccess) return (int)e;
  ++s->open;
  *beside = s->beside;
  return 0;
}

KVB_EXPORT int kvb_side_join(cudaStream_t stream) {
  std::lock_guard<std::mutex> hold(side::guard());
  cudaError_t e = cudaSuccess;
  side::Side* s = side::find(stream, false, e);
  if (s == nullptr) return (int)e;
  --s->open;
  if ((e = cudaEventRecord(s->join, s->beside)) != cudaSuccess) return (int)e;
  return (int)cudaStreamWaitEvent(stream, s->join, 0);
}
