// What a call needs for a moment and the library keeps: pinned staging for host arrays on their way to the device, and events.
//
// Page-locked memory costs a driver call to get, so buffers are kept: per device and power-of-two size at most kKept of
// them (eight of 1 MiB and more, two of 16 MiB and more), each free again when the copy that last read it has finished. When all of a size
// are busy the call waits for the one that has been busy longest.

#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace rlt {
namespace {

constexpr int kKept = 64;
constexpr int kKeptLarge = 8;
constexpr int kKeptHuge = 2;
constexpr int kSmallest = 16;  // log2 bytes
constexpr int kLargest = 40;
constexpr int kMaxDevices = 64;

struct Pinned {
  void* host = nullptr;
  cudaEvent_t done = nullptr;
};
struct SizeClass {
  std::vector<Pinned> buffers;
  size_t next = 0;  // the one that was handed out longest ago
};

std::mutex g_mutex;

// The buffer for `bytes` bytes on the current device; the caller holds g_mutex.
int acquire(size_t bytes, Pinned** out) {
  static SizeClass classes[kMaxDevices][kLargest + 1];
  int device = 0;
  RLT_CUDA_TRY(cudaGetDevice(&device));
  int log = kSmallest;
  while (log <= kLargest && (size_t{1} << log) < bytes) ++log;
  if (device < 0 || device >= kMaxDevices || log > kLargest) return RLT_E_LIMIT;
  SizeClass& c = classes[device][log];
  const size_t kept = log >= 24 ? kKeptHuge : log >= 20 ? kKeptLarge : kKept;
  if (!c.buffers.empty()) {
    Pinned& oldest = c.buffers[c.next];
    const cudaError_t state = cudaEventQuery(oldest.done);
    if (state != cudaSuccess && state != cudaErrorNotReady) return cuda_fail(state);
    if (state == cudaErrorNotReady) cudaGetLastError();  // "not ready" is an answer, not an error to leave behind
    if (state == cudaSuccess || c.buffers.size() >= kept) {
      if (state != cudaSuccess) RLT_CUDA_TRY(cudaEventSynchronize(oldest.done));
      c.next = (c.next + 1) % c.buffers.size();
      *out = &oldest;
      return RLT_OK;
    }
  }
  Pinned fresh;
  RLT_CUDA_TRY(cudaHostAlloc(&fresh.host, size_t{1} << log, cudaHostAllocDefault));
  if (const cudaError_t e = cudaEventCreateWithFlags(&fresh.done, cudaEventDisableTiming); e != cudaSuccess) {
    cudaFreeHost(fresh.host);
    return cuda_fail(e);
  }
  // it takes the place just before the oldest: handed out now, it comes round last
  c.buffers.insert(c.buffers.begin() + static_cast<std::ptrdiff_t>(c.next), fresh);
  *out = &c.buffers[c.next];
  c.next = (c.next + 1) % c.buffers.size();
  return RLT_OK;
}

constexpr size_t kPooledEvents = 256;  // per device and kind; more than that are destroyed when given back
std::mutex g_event_mutex;
std::vector<cudaEvent_t> g_events[kMaxDevices][2];

}  // namespace
}  // namespace rlt

struct RltEvent {
  cudaEvent_t event;
  int device, timed;
};

extern "C" int rlt_event_record(int timed, rlt_stream_t stream, RltEvent** out) {
  int device = 0;
  RLT_CUDA_TRY(cudaGetDevice(&device));
  if (device < 0 || device >= rlt::kMaxDevices) return RLT_E_LIMIT;
  cudaEvent_t event = nullptr;
  {
    const std::lock_guard<std::mutex> lock(rlt::g_event_mutex);
    auto& pool = rlt::g_events[device][timed != 0];
    if (!pool.empty()) {
      event = pool.back();
      pool.pop_back();
    }
  }
  if (event == nullptr) RLT_CUDA_TRY(cudaEventCreateWithFlags(&event, timed ? cudaEventDefault : cudaEventDisableTiming));
  if (const cudaError_t e = cudaEventRecord(event, reinterpret_cast<cudaStream_t>(stream)); e != cudaSuccess) {
    cudaEventDestroy(event);
    return rlt::cuda_fail(e);
  }
  *out = new RltEvent{event, device, timed != 0};
  return RLT_OK;
}

extern "C" int rlt_event_query(RltEvent* event) {
  const cudaError_t e = cudaEventQuery(event->event);
  if (e == cudaSuccess) return 1;
  if (e != cudaErrorNotReady) return rlt::cuda_fail(e);
  cudaGetLastError();  // "not ready" is an answer, not an error to leave behind
  return 0;
}

extern "C" int rlt_event_wait(RltEvent* event) {
  RLT_CUDA_TRY(cudaEventSynchronize(event->event));
  return RLT_OK;
}

extern "C" int rlt_event_elapsed(RltEvent* from, RltEvent* to, float* milliseconds) {
  RLT_CUDA_TRY(cudaEventElapsedTime(milliseconds, from->event, to->event));
  return RLT_OK;
}

extern "C" void rlt_event_release(RltEvent* event) {
  {
    const std::lock_guard<std::mutex> lock(rlt::g_event_mutex);
    auto& pool = rlt::g_events[event->device][event->timed];
    if (pool.size() < rlt::kPooledEvents) {
      pool.push_back(event->event);
      event->event = nullptr;
    }
  }
  if (event->event != nullptr) cudaEventDestroy(event->event);
  delete event;
}

extern "C" int rlt_stage_upload(const void* host, size_t bytes, void* device, rlt_stream_t stream) {
  if (bytes == 0) return RLT_OK;
  if (host == nullptr || device == nullptr) return RLT_E_INVALID;
  const std::lock_guard<std::mutex> lock(rlt::g_mutex);
  rlt::Pinned* slot = nullptr;
  const int rc = rlt::acquire(bytes, &slot);
  if (rc != RLT_OK) return rc;
  std::memcpy(slot->host, host, bytes);
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  RLT_CUDA_TRY(cudaMemcpyAsync(device, slot->host, bytes, cudaMemcpyHostToDevice, s));
  RLT_CUDA_TRY(cudaEventRecord(slot->done, s));
  return RLT_OK;
}
