// Library-wide state and the information entry points.
#include "common.cuh"
#include "internal.h"

namespace rlt {

thread_local int g_last_cuda_error = 0;
std::atomic<long long> g_launches{0};

int sm_count(int* out) {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices];
  int device = 0;
  RLT_CUDA_TRY(cudaGetDevice(&device));
  if (device < 0 || device >= kMaxDevices) return RLT_E_LIMIT;
  int n = cached[device].load(std::memory_order_relaxed);
  if (n == 0) {
    RLT_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device));
    cached[device].store(n, std::memory_order_relaxed);
  }
  *out = n;
  return RLT_OK;
}

std::atomic<long long> g_asking{0}, g_lookups{0};

namespace {

bool own(const void* at) {
  g_lookups.fetch_add(1, std::memory_order_relaxed);
  cudaPointerAttributes of = {};
  int device = -1;
  if (cudaPointerGetAttributes(&of, at) != cudaSuccess || cudaGetDevice(&device) != cudaSuccess) {
    cudaGetLastError();  // an address that nobody knows is no error here
    return false;
  }
  return of.type == cudaMemoryTypeDevice && of.device == device;
}

// The allocation that holds an address; false where the driver does not say.
bool allocation_of(uintptr_t at, unsigned long long* base, size_t* size) {
  using GetRange = int (*)(unsigned long long*, size_t*, unsigned long long);
  static const GetRange get = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<GetRange>(fn);
  }();
  return get != nullptr && get(base, size, at) == 0 && *base <= at && at - *base < *size;
}

}  // namespace

bool prefetches(const void* src, long long bytes) { return bytes >= kPrefetchBytes && own(src); }

bool OwnMemory::holds(const void* from, long long bytes) {
  uintptr_t at = reinterpret_cast<uintptr_t>(from);
  const uintptr_t end = at + static_cast<uintptr_t>(bytes);
  const auto in = [&](int k) { return known_[k].begin <= at && at < known_[k].end; };
  while (at < end) {
    if (last_ >= count_ || !in(last_)) {
      for (last_ = 0; last_ < count_ && !in(last_); ++last_) {
      }
    }
    if (last_ == count_) {
      unsigned long long base = 0;
      size_t size = 0;
      if (count_ == kLookups || !own(reinterpret_cast<const void*>(at)) || !allocation_of(at, &base, &size)) return false;
      known_[count_++] = {static_cast<uintptr_t>(base), static_cast<uintptr_t>(base) + size};
    }
    at = known_[last_].end;
  }
  return true;
}

}  // namespace rlt

extern "C" {

int rlt_version(void) { return 1; }

const char* rlt_error_string(int code) {
  switch (code) {
    case RLT_OK: return "ok";
    case RLT_E_INVALID: return "invalid argument";
    case RLT_E_GEOMETRY: return "pool geometry is not dense or differs between source and destination";
    case RLT_E_LIMIT: return "size limit of the entry point exceeded";
    case RLT_E_CUDA: return "CUDA runtime call failed";
    case RLT_E_ALIGN: return "pointer or size is not aligned as the entry point requires";
    default: return "unknown error";
  }
}

int rlt_last_cuda_error(void) { return rlt::g_last_cuda_error; }

void rlt_prefetch_counts(int64_t counts[2]) {
  counts[0] = rlt::g_asking.load(std::memory_order_relaxed);
  counts[1] = rlt::g_lookups.load(std::memory_order_relaxed);
}

int64_t rlt_kernel_launches(void) { return rlt::g_launches.load(std::memory_order_relaxed); }

}  // extern "C"
