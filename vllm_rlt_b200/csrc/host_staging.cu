// What a call needs for a moment and the library keeps: pinned staging for host arrays on their way to the device, and events.
//
// Page-locked memory costs a driver call to get, so buffers are kept: per device and power-of-two size at most kKept of
// them (eight of 1 MiB and more, two of 16 MiB and more), each free again when the copy that last read it has finished. When all of a
// size are busy the call waits for the one that has been busy longest.

#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "slot_pool.h"

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

int make_pinned(size_t bytes, Pinned* out) {
  Pinned fresh;
  RLT_CUDA_TRY(cudaHostAlloc(&fresh.host, bytes, cudaHostAllocDefault));
  if (const cudaError_t e = cudaEventCreateWithFlags(&fresh.done, cudaEventDisableTiming); e != cudaSuccess) {
    cudaFreeHost(fresh.host);
    return cuda_fail(e);
  }
  *out = fresh;
  return RLT_OK;
}

// Size class of `bytes` on the current device.
struct PinnedClass {
  SlotPool<Pinned>* pool;
  size_t bytes, kept;
};
int pinned_class(size_t bytes, PinnedClass* out) {
  static auto* pools = new SlotPool<Pinned>[kMaxDevices][kLargest + 1];  // never destroyed: threads may outlive main
  int device = 0;
  RLT_CUDA_TRY(cudaGetDevice(&device));
  int log = kSmallest;
  while (log <= kLargest && (size_t{1} << log) < bytes) ++log;
  if (device < 0 || device >= kMaxDevices || log > kLargest) return RLT_E_LIMIT;
  *out = {&pools[device][log], size_t{1} << log, static_cast<size_t>(log >= 24 ? kKeptHuge : log >= 20 ? kKeptLarge : kKept)};
  return RLT_OK;
}

// Buffers that captured copies read: a replay may come at any time, so they are the graph's until it is destroyed. Then they are kept
// for later captures, as many as were in graphs at once: the runtime allows no call of its own, like one that frees memory, where it
// tells of a graph's end.
struct GraphBuffers {
  std::mutex mutex;
  std::vector<void*> idle;
};
GraphBuffers& graph_buffers(int log) {
  static auto* all = new GraphBuffers[kLargest + 1];
  return all[log];
}
struct GraphBuffer {
  void* host;
  int log;
};
void graph_is_gone(void* p) {
  auto* buffer = static_cast<GraphBuffer*>(p);
  GraphBuffers& of = graph_buffers(buffer->log);
  {
    const std::lock_guard<std::mutex> lock(of.mutex);
    of.idle.push_back(buffer->host);
  }
  delete buffer;
}

int upload_in_capture(const void* host, size_t bytes, void* device, cudaStream_t stream, cudaGraph_t graph) {
  int log = kSmallest;
  while (log <= kLargest && (size_t{1} << log) < bytes) ++log;
  if (log > kLargest) return RLT_E_LIMIT;
  auto* buffer = new GraphBuffer{nullptr, log};
  GraphBuffers& of = graph_buffers(log);
  {
    const std::lock_guard<std::mutex> lock(of.mutex);
    if (!of.idle.empty()) {
      buffer->host = of.idle.back();
      of.idle.pop_back();
    }
  }
  const OutsideCapture outside;
  cudaError_t e = cudaSuccess;
  // portable: graphs of another device may get it after this one
  if (buffer->host == nullptr) e = cudaHostAlloc(&buffer->host, size_t{1} << log, cudaHostAllocPortable);
  cudaUserObject_t owner = nullptr;
  if (e == cudaSuccess) {
    std::memcpy(buffer->host, host, bytes);
    e = cudaUserObjectCreate(&owner, buffer, graph_is_gone, 1, cudaUserObjectNoDestructorSync);
  }
  if (e != cudaSuccess) {
    if (buffer->host != nullptr) {
      graph_is_gone(buffer);
    } else {
      delete buffer;
    }
    return cuda_fail(e);
  }
  e = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(owner, 1);
    return cuda_fail(e);
  }
  RLT_CUDA_TRY(cudaMemcpyAsync(device, buffer->host, bytes, cudaMemcpyHostToDevice, stream));
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
  const rlt::OutsideCapture outside;
  if (event == nullptr) RLT_CUDA_TRY(cudaEventCreateWithFlags(&event, timed ? cudaEventDefault : cudaEventDisableTiming));
  if (const cudaError_t e = cudaEventRecord(event, reinterpret_cast<cudaStream_t>(stream)); e != cudaSuccess) {
    cudaEventDestroy(event);
    return rlt::cuda_fail(e);
  }
  *out = new RltEvent{event, device, timed != 0};
  return RLT_OK;
}

extern "C" int rlt_event_query(RltEvent* event) {
  const rlt::OutsideCapture outside;
  const cudaError_t e = cudaEventQuery(event->event);
  if (e == cudaSuccess) return 1;
  if (e != cudaErrorNotReady) return rlt::cuda_fail(e);
  cudaGetLastError();  // "not ready" is an answer, not an error to leave behind
  return 0;
}

extern "C" int rlt_event_wait(RltEvent* event) {
  const rlt::OutsideCapture outside;
  RLT_CUDA_TRY(cudaEventSynchronize(event->event));
  return RLT_OK;
}

extern "C" int rlt_event_order(RltEvent* event, rlt_stream_t stream) {
  RLT_CUDA_TRY(cudaStreamWaitEvent(reinterpret_cast<cudaStream_t>(stream), event->event, 0));
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
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  RLT_CUDA_TRY(cudaStreamGetCaptureInfo(s, &capturing, nullptr, &graph));
  if (capturing != cudaStreamCaptureStatusNone) return rlt::upload_in_capture(host, bytes, device, s, graph);
  rlt::PinnedClass size;
  int rc = rlt::pinned_class(bytes, &size);
  if (rc != RLT_OK) return rc;
  rlt::Pinned slot;
  rc = size.pool->take(&slot, size.kept, [&](rlt::Pinned* fresh) { return rlt::make_pinned(size.bytes, fresh); });
  if (rc != RLT_OK) return rc;
  std::memcpy(slot.host, host, bytes);
  cudaError_t e = cudaMemcpyAsync(device, slot.host, bytes, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaEventRecord(slot.done, s);
  size.pool->give(slot);
  RLT_CUDA_TRY(e);
  return RLT_OK;
}

extern "C" int rlt_capture_id(rlt_stream_t stream, uint64_t* id) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  unsigned long long of = 0;
  RLT_CUDA_TRY(cudaStreamGetCaptureInfo(reinterpret_cast<cudaStream_t>(stream), &capturing, &of));
  *id = capturing == cudaStreamCaptureStatusNone ? 0 : of;
  return RLT_OK;
}
