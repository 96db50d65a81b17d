// Shared host/device helpers of the KV-handoff kernels (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <nvtx3/nvToolsExt.h>

#include <atomic>

#include "rlt_kv_handoff.h"

namespace rlt {

constexpr int kThreads = 256;      // threads per CTA of every copy kernel
constexpr int kMaxRows = 256;      // token rows one work unit may hold
constexpr int kMaxBlockSize = 64;  // tokens per KV block

extern thread_local int g_last_cuda_error;
extern std::atomic<long long> g_launches;

inline int cuda_fail(cudaError_t e) {
  g_last_cuda_error = static_cast<int>(e);
  return RLT_E_CUDA;
}

#define RLT_CUDA_TRY(expr)                          \
  do {                                              \
    cudaError_t rlt_err__ = (expr);                 \
    if (rlt_err__ != cudaSuccess) return ::rlt::cuda_fail(rlt_err__); \
  } while (0)

// Names the launches of one entry point for profilers (the reference's NIXL traffic is invisible to its
// torch profiler sessions; these launches are ordinary kernels and show up under these ranges).
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// SM count of the current device, looked up once per device.
int sm_count(int* out);

// Launch that may be set up while the kernel before it on the stream is finishing (programmatic stream serialisation). The
// kernel calls follow_stream() before it touches any memory but its parameters: that returns when everything before it on the
// stream has completed and is visible, and then lets the next such launch be set up behind this one. Saves most of the gap
// between two short kernels; kernels launched the ordinary way, copies and events are ordered as ever.
// What such a kernel reads may still be written by the one before it while it is being set up, so none of its pointers is __restrict__: that
// would promise the compiler memory that nobody writes for as long as the kernel runs, and let it read ahead of the wait or through a cache
// that is not coherent.
template <typename T>
struct Given {  // the type of the parameter, whatever is given for it
  using type = T;
};
template <typename... P>
inline cudaError_t launch_following(void (*kernel)(P...), dim3 grid, unsigned block, cudaStream_t stream, const typename Given<P>::type&... args) {
  cudaLaunchAttribute attribute = {};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(block);
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  // by address: the typed form of the call copies the parameters once more first (0.6 us of a launch's 3.7 where they are 31 KB)
  void* at[] = {const_cast<void*>(static_cast<const void*>(&args))...};
  return cudaLaunchKernelExC(&config, reinterpret_cast<const void*>(kernel), at);
}
// Loads a kernel, if that has not been done.
template <typename... P>
inline cudaError_t load_kernel(void (*kernel)(P...)) {
  cudaFuncAttributes unused;
  return cudaFuncGetAttributes(&unused, kernel);
}
__device__ __forceinline__ void follow_stream() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Asks L2 for [from, from + bytes), both multiples of 16: nobody waits for it. A kernel launched as above may ask for what it is going to
// read before follow_stream(), while the kernel ahead of it finishes and memory falls idle: what that one still writes it writes to
// L2 as well, so nothing stale is ever read. Only for memory of this GPU: another GPU's would cross the link and not be kept.
__device__ __forceinline__ void prefetch_l2(const char* from, int bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"(bytes) : "memory");
}
// CTAs ahead of its own that a CTA asks for the source of, where that is worked out from the kernel's parameters alone. It keeps reads coming in
// the moment between a CTA's end and the next one's first load. Copies of 32 MiB - 1 GiB in 16 KiB pieces, TB/s without / own piece /
// 148, 296 and 592 CTAs ahead as well: 5.82 / 6.36 / 6.65, 6.64, 6.55; 6.71 / 6.79 / 6.82, 6.77, 6.60; 6.87 / 6.92 / 6.89, 6.86, 6.68.
// With the records of block_moves.cu 74 is as good or better than 148 in every case tried (1 GB of FP8 pages: 1,101 / 1,090 / 1,086 us
// at none, own, 74; 1,087 at 148, 1,107 at 592).
constexpr unsigned kPrefetchAhead = 74;
// Bytes that a launch reads and writes from which on it asks. Below that all of them may well be in L2 since they were last used, where asking
// costs a little and gains nothing. us without / with, three pairs of buffers in turn: 24 MB float32 -> bfloat16 3.04 / 3.14, a layer
// slice of 26 MB 4.19 / 4.42 and of 32 MB 5.70 / 5.71; 42 MB 8.8 / 8.0, 48 MB int64 -> int32 8.45 / 7.07, 1.2 GB 172 / 169.
constexpr long long kPrefetchBytes = 32 << 20;
// Whether a launch that moves so many bytes asks for its source, which has to be in memory of the current device (0.07 us to find out).
bool prefetches(const void* src, long long bytes);

// Which addresses are in memory of the current device. An allocation is looked up once, and a few at most: where ranges lie in more of them than
// a worker's pools have tensors, the answer is no.
class OwnMemory {
 public:
  bool holds(const void* from, long long bytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(from), size = static_cast<uintptr_t>(bytes);
    for (int k = 0; k < count_; ++k) {
      if (at - known_[k].begin < known_[k].size && size <= known_[k].size - (at - known_[k].begin)) return true;
    }
    return look_up(at, size);
  }

 private:
  static constexpr int kLookups = 8;
  bool look_up(uintptr_t at, uintptr_t size);
  struct {
    uintptr_t begin, size;
  } known_[kLookups];
  int count_ = 0;
};

// Counts the launches that ask, for the tests.
extern std::atomic<long long> g_asking, g_lookups;
inline bool asking(bool yes) {
  if (yes) g_asking.fetch_add(1, std::memory_order_relaxed);
  return yes;
}

// First error wins: later reports leave the status words alone.
__device__ __forceinline__ void report(int32_t* status, int code, int a, int b, int c) {
  if (status == nullptr) return;
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = a;
    status[2] = b;
    status[3] = c;
  }
}

// Streaming 16-byte accesses: the payload is touched once, keep it out of L1.
__device__ __forceinline__ uint4 ld_stream(const uint4* p) { return __ldcs(p); }
__device__ __forceinline__ void st_stream(uint4* p, uint4 v) { __stcs(p, v); }
// 32-byte accesses (256-bit global loads and stores exist from sm_100 on).
struct alignas(32) Vec32 {
  uint32_t v[8];
};
__device__ __forceinline__ Vec32 ld_stream(const Vec32* p) {
  Vec32 r;
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
                 "=r"(r.v[7])
               : "l"(p));
  return r;
}
__device__ __forceinline__ void st_stream(Vec32* p, const Vec32& r) {
  asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r.v[0]), "r"(r.v[1]),
               "r"(r.v[2]), "r"(r.v[3]), "r"(r.v[4]), "r"(r.v[5]), "r"(r.v[6]), "r"(r.v[7])
               : "memory");
}
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* p) { return __ldcs(p); }
__device__ __forceinline__ void st_stream(uint32_t* p, uint32_t v) { __stcs(p, v); }
__device__ __forceinline__ uint8_t ld_stream(const uint8_t* p) { return *p; }
__device__ __forceinline__ void st_stream(uint8_t* p, uint8_t v) { *p = v; }

// A CTA copies elements [0, n).
template <typename T, int kUnroll = 4>
__device__ __forceinline__ void stream_range(const char* src, char* dst, long long n) {
  const T* s = reinterpret_cast<const T*>(src);
  T* d = reinterpret_cast<T*>(dst);
  for (long long base = threadIdx.x; base < n; base += kThreads * kUnroll) {
    T regs[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long i = base + u * kThreads;
      if (i < n) regs[u] = ld_stream(s + i);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long i = base + u * kThreads;
      if (i < n) st_stream(d + i, regs[u]);
    }
  }
}

// A CTA copies one tile of a byte range. kWide: 32-byte accesses where both pointers allow. Pointers that are both 16-byte
// aligned take the vector path with a byte tail; otherwise the widest element both pointers and the length allow.
template <bool kWide>
__device__ __forceinline__ void copy_piece(const char* src, char* dst, long long n) {
  const unsigned long long both = reinterpret_cast<unsigned long long>(src) | reinterpret_cast<unsigned long long>(dst);
  if (kWide && (both & 31ull) == 0) {
    const long long body = n & ~31ll;
    stream_range<Vec32, 2>(src, dst, body >> 5);
    if (static_cast<long long>(threadIdx.x) < n - body) dst[body + threadIdx.x] = src[body + threadIdx.x];
  } else if ((both & 15ull) == 0) {
    const long long body = n & ~15ll;
    stream_range<uint4>(src, dst, body >> 4);
    if (static_cast<long long>(threadIdx.x) < n - body) dst[body + threadIdx.x] = src[body + threadIdx.x];
  } else if (((both | static_cast<unsigned long long>(n)) & 3ull) == 0) {
    stream_range<uint32_t>(src, dst, n >> 2);
  } else {
    stream_range<uint8_t>(src, dst, n);
  }
}

// Inclusive prefix sum across the 32 lanes of a warp.
__device__ __forceinline__ int warp_inclusive_scan(int v) {
  const unsigned lane = threadIdx.x & 31u;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int n = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= static_cast<unsigned>(d)) v += n;
  }
  return v;
}

// Multiplier m with floor(i / d) == __umulhi(i, m) whenever i * d < 2^32.
inline uint32_t div_magic(uint32_t d) { return static_cast<uint32_t>((1ull << 32) / d) + 1u; }

}  // namespace rlt
