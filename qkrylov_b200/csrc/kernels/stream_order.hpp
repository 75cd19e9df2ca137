// Order of a plan's calls across streams.
//
// The row, spin-product and block kernels keep state in their plan between a
// launch's blocks: work-queue counters, partial sums, the product-ordered
// scratch.  Two launches of one plan must therefore not overlap.  On one stream
// they cannot; when a call names another stream than the call before it, that
// stream first waits for the earlier call.
//
// The home stream (the library's, which outlives every plan) costs nothing: its
// event is recorded only when another stream follows.  A caller's stream may be
// gone by then, so there the event is recorded after every call.
#pragma once

#include <mutex>

#include <cuda_runtime.h>

namespace qkd {

class StreamOrder {
 public:
  explicit StreamOrder(cudaStream_t home) : home_(home) {}
  ~StreamOrder() {
    if (ev_) cudaEventDestroy(ev_);
  }
  StreamOrder(const StreamOrder&) = delete;
  StreamOrder& operator=(const StreamOrder&) = delete;

  bool init() { return cudaEventCreateWithFlags(&ev_, cudaEventDisableTiming) == cudaSuccess; }

  // Held over the launches of one call on stream s, which keeps host threads
  // apart as well.  A call in capture is ordered by its graph alone.
  class Use {
   public:
    Use(StreamOrder& o, cudaStream_t s) : o_(o), lk_(o.mu_), s_(s) {
      if (capturing(s) || cudaStreamGetId(s, &id_) != cudaSuccess) {
        (void)cudaGetLastError();
        return;
      }
      live_ = true;
      if (!o_.any_ || o_.last_ == id_) return;
      if (o_.at_home_ && (capturing(o_.home_) || cudaEventRecord(o_.ev_, o_.home_) != cudaSuccess)) {
        (void)cudaGetLastError();
        return;
      }
      if (cudaStreamWaitEvent(s, o_.ev_, 0) != cudaSuccess) (void)cudaGetLastError();
    }
    ~Use() {
      if (!live_) return;
      o_.any_ = true;
      o_.last_ = id_;
      o_.at_home_ = s_ == o_.home_;
      if (!o_.at_home_ && cudaEventRecord(o_.ev_, s_) != cudaSuccess) (void)cudaGetLastError();
    }
    Use(const Use&) = delete;
    Use& operator=(const Use&) = delete;

   private:
    static bool capturing(cudaStream_t s) {
      cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
      return cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone;
    }
    StreamOrder& o_;
    std::lock_guard<std::mutex> lk_;
    cudaStream_t s_;
    unsigned long long id_ = 0;
    bool live_ = false;
  };

 private:
  std::mutex mu_;
  cudaStream_t home_;
  cudaEvent_t ev_ = nullptr;
  unsigned long long last_ = 0;  // id of the last call's stream (handles are reused, ids are not)
  bool any_ = false, at_home_ = false;
};

}  // namespace qkd
