// Host memory that the GPU reads later, handed out in turn: what the staging of host_staging.cu and kv_table_copy.cu share.
#pragma once

#include <cuda_runtime.h>

#include <condition_variable>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace rlt {

// Lets the thread make calls that are not allowed while a stream is capturing a graph, about things that the capture has no part in.
struct OutsideCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// `Slot` has a `done` event, recorded behind the last work that reads the slot. A slot belongs to the thread that took it until it
// gives it back, so nothing is locked while that thread fills it, queues the work, or waits for the GPU to let go of it.
template <typename Slot>
class SlotPool {
 public:
  // A slot that nothing reads any more. The one given back longest ago whose work is over; if there is none, a fresh one from
  // `make(Slot*)` while fewer than `most` exist; else the one given back longest ago, once its work is over.
  template <typename Make>
  int take(Slot* out, size_t most, Make make) {
    const OutsideCapture outside;
    std::unique_lock<std::mutex> lock(mutex_);
    for (;;) {
      for (auto it = idle_.begin(); it != idle_.end(); ++it) {
        const cudaError_t state = cudaEventQuery(it->done);
        if (state == cudaSuccess) {
          *out = *it;
          idle_.erase(it);
          return RLT_OK;
        }
        if (state != cudaErrorNotReady) return cuda_fail(state);
        cudaGetLastError();  // "not ready" is an answer, not an error to leave behind
      }
      if (count_ < most) {
        ++count_;
        lock.unlock();
        const int rc = make(out);
        if (rc == RLT_OK) return RLT_OK;
        lock.lock();
        --count_;
        returned_.notify_one();  // a thread that counted on this slot looks again
        return rc;
      }
      if (!idle_.empty()) {
        *out = idle_.front();
        idle_.erase(idle_.begin());
        lock.unlock();
        const cudaError_t state = cudaEventSynchronize(out->done);
        if (state == cudaSuccess) return RLT_OK;
        give(*out);
        return cuda_fail(state);
      }
      returned_.wait(lock);  // other threads are filling all of them
    }
  }
  void give(const Slot& slot) {
    {
      const std::lock_guard<std::mutex> lock(mutex_);
      idle_.push_back(slot);
    }
    returned_.notify_one();
  }

 private:
  std::mutex mutex_;
  std::condition_variable returned_;
  std::vector<Slot> idle_;  // given back longest ago first
  size_t count_ = 0;        // that exist, idle or taken
};

}  // namespace rlt
