// Completion flags between the prefill GPU and the decode GPU.
//
// The reference learns that a chunk has landed from the notification NIXL
// delivers with each WRITE (vllm_rlt/pd/transport.py:186-195, :222-229). Here
// the sender issues a release store on the stream that carried the copy, and
// the receiver either polls the word from the host or runs the bounded wait
// below ahead of the work that consumes the KV.
//
// The wait never spins without a limit: it watches %globaltimer and gives up
// after the caller's timeout, recording what it last saw.

#include <cstring>

#include "block_moves.h"
#include "common.cuh"
#include "internal.h"

namespace rlt {
namespace {

__global__ void signal_kernel(unsigned long long* flag, unsigned long long value) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    __threadfence_system();
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(flag), "l"(value) : "memory");
  }
}

// A mailbox message: a body of seven words, then the stamp. One thread copies nothing but these; a block first copies the small ranges that
// ride on the message (a hidden-state row), which spares a launch of their own.
//
// Bound by latency: the launch, and a write to host memory behind a system-wide fence. Launched as launch_following does, so that the launch
// and the end of the copy before it overlap, and with the release as the only fence, it adds 3.2 us to a copy of 0.5 GB on one B200;
// launched the ordinary way with a second fence before the release it was 6.4. (The message as the last act of the copy's own last block adds
// 6 - 8: every block then has to wait for its writes.)
struct PostArgs {
  unsigned long long* slot;
  unsigned long long words[7];
  unsigned long long stamp;
  int ranges;
  const char* src[RLT_POST_RANGES];
  char* dst[RLT_POST_RANGES];
  long long bytes[RLT_POST_RANGES];
};

__global__ void post_kernel(const __grid_constant__ PostArgs a) {
  follow_stream();
  if (a.ranges > 0) {
#pragma unroll 1
    for (int i = 0; i < a.ranges; ++i) copy_piece<true>(a.src[i], a.dst[i], a.bytes[i]);
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
#pragma unroll
  for (int i = 0; i < 7; ++i) a.slot[1 + i] = a.words[i];
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(a.slot), "l"(a.stamp) : "memory");
}

__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__global__ void wait_kernel(const unsigned long long* flag, unsigned long long value, long long timeout_ns,
                            int* status) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const unsigned long long start = global_timer_ns();
  unsigned long long seen = 0;
  // Two limits: elapsed time, and an iteration cap in case the timer does not advance.
  for (long long spin = 0; spin < (1ll << 34); ++spin) {
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(seen) : "l"(flag) : "memory");
    if (seen >= value) return;
    if (global_timer_ns() - start > static_cast<unsigned long long>(timeout_ns)) break;
    __nanosleep(200);
  }
  report(status, RLT_STATUS_TIMEOUT, static_cast<int>(seen & 0xffffffffull), 0, 0);
}

}  // namespace
}  // namespace rlt

extern "C" {

int rlt_kv_signal(uint64_t* flag, uint64_t value, rlt_stream_t stream) {
  if (flag == nullptr) return RLT_E_INVALID;
  if (reinterpret_cast<uintptr_t>(flag) & 7u) return RLT_E_ALIGN;
  rlt::signal_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<unsigned long long*>(flag), value);
  RLT_CUDA_TRY(cudaGetLastError());
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

int rlt_kv_post(void* slot, const uint8_t body[56], uint64_t stamp, rlt_stream_t stream) {
  return rlt_post_behind(nullptr, 0, slot, body, stamp, stream);
}

int rlt_post_behind(const int64_t* ranges, int32_t count, void* slot, const uint8_t body[56], uint64_t stamp, rlt_stream_t stream) {
  if (slot == nullptr || body == nullptr) return RLT_E_INVALID;
  if (reinterpret_cast<uintptr_t>(slot) & 15u) return RLT_E_ALIGN;
  if (count < 0 || (count > 0 && ranges == nullptr)) return RLT_E_INVALID;
  if (count > RLT_POST_RANGES) return RLT_E_LIMIT;
  rlt::PostArgs a = {};
  a.slot = static_cast<unsigned long long*>(slot);
  std::memcpy(a.words, body, sizeof(a.words));
  a.stamp = stamp;
  a.ranges = count;
  int64_t bytes = 0;
  for (int i = 0; i < count; ++i) {
    a.src[i] = reinterpret_cast<const char*>(ranges[3 * i]);
    a.dst[i] = reinterpret_cast<char*>(ranges[3 * i + 1]);
    a.bytes[i] = ranges[3 * i + 2];
    if (a.bytes[i] < 0 || (a.bytes[i] > 0 && (a.src[i] == nullptr || a.dst[i] == nullptr))) return RLT_E_INVALID;
    if (a.bytes[i] > RLT_POST_RANGE_BYTES - bytes) return RLT_E_LIMIT;
    bytes += a.bytes[i];
  }
  RLT_CUDA_TRY(rlt::launch_following(rlt::post_kernel, 1, count > 0 ? rlt::kThreads : 32, reinterpret_cast<cudaStream_t>(stream), a));
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

int rlt_load_transport(int32_t planes) {
  RLT_CUDA_TRY(rlt::load_kernel(rlt::post_kernel));
  const int rc = rlt_load_segments();
  if (rc != RLT_OK) return rc;
  // The table-driven kernels bring 4.2 MB of device memory with them, so only for the pools that need them; where that does not fit, the first
  // launch will say so.
  if (planes > kMaxRecordPlanes && rlt_load_tables() != RLT_OK) (void)cudaGetLastError();
  return rlt_load_moves();
}

int rlt_kv_wait(const uint64_t* flag, uint64_t value, int64_t timeout_ns, int32_t* status, rlt_stream_t stream) {
  if (flag == nullptr || status == nullptr) return RLT_E_INVALID;
  if (reinterpret_cast<uintptr_t>(flag) & 7u) return RLT_E_ALIGN;
  if (timeout_ns < 1 || timeout_ns > RLT_MAX_WAIT_NS) return RLT_E_LIMIT;
  rlt::wait_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const unsigned long long*>(flag), value, timeout_ns, status);
  RLT_CUDA_TRY(cudaGetLastError());
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

}  // extern "C"
