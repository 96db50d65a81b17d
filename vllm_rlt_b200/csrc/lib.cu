// Library-wide state and the information entry points.
#include <cuda.h>

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

bool prefetches(const void* src, long long bytes) {
  if (bytes < kPrefetchBytes) return false;
  g_lookups.fetch_add(1, std::memory_order_relaxed);
  cudaPointerAttributes of = {};
  int device = -1;
  if (cudaPointerGetAttributes(&of, src) != cudaSuccess || cudaGetDevice(&device) != cudaSuccess) {
    cudaGetLastError();  // an address that nobody knows is no error here
    return false;
  }
  return of.type == cudaMemoryTypeDevice && of.device == device;
}

// The allocation that holds an address, if it is memory of the current device. One call of the driver's (0.06 us) where the runtime would take two.
static bool own_allocation(uintptr_t at, uintptr_t* begin, uintptr_t* size) {
  using Attributes = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
  static const Attributes ask = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &fn, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<Attributes>(fn);
  }();
  g_lookups.fetch_add(1, std::memory_order_relaxed);
  unsigned type = 0, managed = 0;  // (the driver writes four bytes for either)
  int of = -1, device = -2;
  CUdeviceptr base = 0;
  size_t bytes = 0;
  CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* where[] = {&type, &of, &managed, &base, &bytes};
  if (ask == nullptr || ask(5, what, where, at) != CUDA_SUCCESS || cudaGetDevice(&device) != cudaSuccess) return false;
  *begin = base;
  *size = bytes;
  return type == CU_MEMORYTYPE_DEVICE && managed == 0 && of == device && base <= at && at - base < bytes;
}

bool OwnMemory::look_up(uintptr_t at, uintptr_t size) {
  for (const uintptr_t end = at + size; at < end;) {
    int k = 0;
    while (k < count_ && at - known_[k].begin >= known_[k].size) ++k;
    if (k == count_) {
      if (count_ == kLookups || !own_allocation(at, &known_[k].begin, &known_[k].size)) return false;
      ++count_;
    }
    at = known_[k].begin + known_[k].size;
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
