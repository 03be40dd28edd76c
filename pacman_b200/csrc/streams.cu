// Idle streams and events of the library, kept per device between calls.
#include <mutex>
#include <vector>

#include "plan.hpp"

namespace pacman_b200 {

namespace {

constexpr int kMaxDevices = 64;
constexpr size_t kMaxIdleStreams = 16;  // a batch takes one per host thread and its own

struct Idle {
  std::mutex mu;
  std::vector<AuxStreams::Set *> sets;
  std::vector<cudaStream_t> streams;
};

// Never destroyed: the CUDA runtime may be gone when statics are.
Idle *idle_of(int device) {
  static Idle *lists = new Idle[kMaxDevices];
  return device >= 0 && device < kMaxDevices ? lists + device : nullptr;
}

void destroy_set(AuxStreams::Set *set) {
  for (cudaStream_t s : set->s)
    if (s) cudaStreamDestroy(s);
  for (cudaEvent_t e : set->ev)
    if (e) cudaEventDestroy(e);
  delete set;
}

}  // namespace

void AuxStreams::make() {
  if (set_) return;
  int device = 0;
  PB_CUDA(cudaGetDevice(&device));
  if (Idle *idle = idle_of(device)) {
    std::lock_guard<std::mutex> lock(idle->mu);
    if (!idle->sets.empty()) {
      set_ = idle->sets.back();
      idle->sets.pop_back();
    }
  }
  if (!set_) {
    Set *set = new Set();
    set->device = device;
    try {
      int least = 0, greatest = 0;
      PB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
      for (int i = 0; i <= kN; ++i)
        PB_CUDA(cudaStreamCreateWithPriority(&set->s[i], cudaStreamNonBlocking,
                                             i == kSmall ? least : greatest));
      for (cudaEvent_t &e : set->ev)
        PB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    } catch (...) {
      destroy_set(set);
      throw;
    }
    set_ = set;
  }
  s = set_->s;
  ev = set_->ev;
}

AuxStreams::~AuxStreams() {
  if (!set_) return;
  if (Idle *idle = idle_of(set_->device)) {
    std::lock_guard<std::mutex> lock(idle->mu);
    if (idle->sets.size() < kMaxIdle) {
      idle->sets.push_back(set_);
      set_ = nullptr;
    }
  }
  if (set_) destroy_set(set_);
}

cudaStream_t take_stream(int device) {
  cudaStream_t s = nullptr;
  if (Idle *idle = idle_of(device)) {
    std::lock_guard<std::mutex> lock(idle->mu);
    if (!idle->streams.empty()) {
      s = idle->streams.back();
      idle->streams.pop_back();
    }
  }
  if (!s) PB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  return s;
}

void order_after(cudaStream_t st, cudaStream_t before) {
  cudaEvent_t e;
  PB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  cudaError_t rc = cudaEventRecord(e, before);
  if (rc == cudaSuccess) rc = cudaStreamWaitEvent(st, e, 0);
  cudaEventDestroy(e);
  PB_CUDA(rc);
}

void await_default_stream(cudaStream_t s) {
  // Not while a capture is under way that the legacy stream would break.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(cudaStreamLegacy, &cap) == cudaSuccess &&
      cap == cudaStreamCaptureStatusNone)
    order_after(s, cudaStreamLegacy);
  cudaGetLastError();
}

void give_stream(cudaStream_t s, int device) {
  if (!s) return;
  const bool ok = cudaStreamSynchronize(s) == cudaSuccess;
  if (Idle *idle = ok ? idle_of(device) : nullptr) {
    std::lock_guard<std::mutex> lock(idle->mu);
    if (idle->streams.size() < kMaxIdleStreams) {
      idle->streams.push_back(s);
      return;
    }
  }
  cudaStreamDestroy(s);
}

}  // namespace pacman_b200
