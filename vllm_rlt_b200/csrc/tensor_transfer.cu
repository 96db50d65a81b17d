// Typed tensor movement: a flat copy with an optional second output of another type, and batches
// of strided 2-D copies described by a table of int64[8] rows
// (source address, destination address, rows, cols, source row/col stride, destination row/col
// stride; strides in elements). It takes the place of the reference's Triton
// tensor_transfer_kernel (vllm_rlt/kernels/tensor_transfer.py:8-42), which moves step metadata,
// block tables and hidden-state rows on one device or from mapped host memory to the device.
//
// Element types are int32, int64, float16, bfloat16 and float32. Values are converted by the
// usual cast rules (integer narrowing wraps, float -> integer truncates toward zero, integer and
// float -> float round to nearest even). Integers never pass through a floating type, so int64
// ids above 2^53 survive an int64 -> int64 copy exactly.

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstring>

#include "common.cuh"
#include "internal.h"

namespace rlt {
namespace {

template <typename D, typename S>
struct Convert {
  __device__ static D run(S v) { return static_cast<D>(v); }
};
// float-like sources go through float; float-like destinations come from float or the integer itself
template <typename D>
struct Convert<D, __half> {
  __device__ static D run(__half v) { return Convert<D, float>::run(__half2float(v)); }
};
template <typename D>
struct Convert<D, __nv_bfloat16> {
  __device__ static D run(__nv_bfloat16 v) { return Convert<D, float>::run(__bfloat162float(v)); }
};
template <>
struct Convert<__half, float> {
  __device__ static __half run(float v) { return __float2half_rn(v); }
};
template <>
struct Convert<__nv_bfloat16, float> {
  __device__ static __nv_bfloat16 run(float v) { return __float2bfloat16_rn(v); }
};
template <>
struct Convert<__half, int> {
  __device__ static __half run(int v) { return __int2half_rn(v); }
};
template <>
struct Convert<__half, long long> {
  __device__ static __half run(long long v) { return __ll2half_rn(v); }
};
template <>
struct Convert<__nv_bfloat16, int> {
  __device__ static __nv_bfloat16 run(int v) { return __int2bfloat16_rn(v); }
};
template <>
struct Convert<__nv_bfloat16, long long> {
  __device__ static __nv_bfloat16 run(long long v) { return __ll2bfloat16_rn(v); }
};
template <>
struct Convert<__half, __half> {
  __device__ static __half run(__half v) { return v; }
};
template <>
struct Convert<__nv_bfloat16, __nv_bfloat16> {
  __device__ static __nv_bfloat16 run(__nv_bfloat16 v) { return v; }
};
template <>
struct Convert<__half, __nv_bfloat16> {
  __device__ static __half run(__nv_bfloat16 v) { return __float2half_rn(__bfloat162float(v)); }
};
template <>
struct Convert<__nv_bfloat16, __half> {
  __device__ static __nv_bfloat16 run(__half v) { return __float2bfloat16_rn(__half2float(v)); }
};

constexpr int kRows = 4;
constexpr int kTile = 256;

template <typename S, typename D>
__global__ void __launch_bounds__(kTile) segmented_transfer_kernel(const long long* descriptors) {
  follow_stream();
  const long long* d = descriptors + 8ll * blockIdx.x;
  const S* src = reinterpret_cast<const S*>(d[0]);
  D* dst = reinterpret_cast<D*>(d[1]);
  const long long rows = d[2], cols = d[3], sr = d[4], sc = d[5], dr = d[6], dc = d[7];
  const long long c = static_cast<long long>(blockIdx.z) * kTile + threadIdx.x;
  if (c >= cols) return;
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const long long r = static_cast<long long>(blockIdx.y) * kRows + k;
    if (r < rows) dst[r * dr + c * dc] = Convert<D, S>::run(src[r * sr + c * sc]);
  }
}

// The same between tensors of one type, whose elements are only moved, with the descriptors in the kernel's parameters: a
// step's handful of small copies waits neither for a table in host memory (a read over PCIe before every copy) nor for
// a host-to-device copy of one. A CTA moves kRows rows of kTileBytes bytes, 16 bytes a thread where both sides are
// contiguous and aligned.
constexpr int kTileBytes = 4096;
constexpr int kInlineSmall = 56;  // descriptors of the smaller parameter block (3.5 KiB)

template <int kCount>
struct InlineDescriptors {
  long long d[kCount][8];
};

template <typename T>
__device__ __forceinline__ void move_tile(const T* src, T* dst, int n, long long sc, long long dc) {
  constexpr int kPer = 16 / sizeof(T);
  const unsigned long long bits = reinterpret_cast<unsigned long long>(src) | reinterpret_cast<unsigned long long>(dst);
  if (sc == 1 && dc == 1 && (bits & 15ull) == 0) {
    const int vectors = n / kPer;
    for (int i = threadIdx.x; i < vectors; i += kTile) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    for (int i = vectors * kPer + threadIdx.x; i < n; i += kTile) dst[i] = src[i];
  } else {
    for (int i = threadIdx.x; i < n; i += kTile) dst[i * dc] = src[i * sc];
  }
}

template <typename T, int kCount>
__global__ void __launch_bounds__(kTile) inline_transfer_kernel(const __grid_constant__ InlineDescriptors<kCount> table) {
  constexpr long long kCols = kTileBytes / static_cast<long long>(sizeof(T));
  const long long* d = table.d[blockIdx.x];
  const long long rows = d[2], cols = d[3], sr = d[4], sc = d[5], dr = d[6], dc = d[7];
  const long long c0 = blockIdx.z * kCols;
  follow_stream();
  if (c0 >= cols) return;
  const int n = static_cast<int>(cols - c0 < kCols ? cols - c0 : kCols);
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const long long r = static_cast<long long>(blockIdx.y) * kRows + k;
    if (r < rows)
      move_tile(reinterpret_cast<const T*>(d[0]) + r * sr + c0 * sc, reinterpret_cast<T*>(d[1]) + r * dr + c0 * dc, n, sc, dc);
  }
}

template <typename T, int kCount>
int launch_inline(const int64_t* descriptors, int count, dim3 grid, cudaStream_t stream) {
  InlineDescriptors<kCount> table;
  std::memcpy(table.d, descriptors, static_cast<size_t>(count) * sizeof(table.d[0]));
  RLT_CUDA_TRY(launch_following(inline_transfer_kernel<T, kCount>, grid, kTile, stream, table));
  return RLT_OK;
}

template <typename T>
int launch_inline(const int64_t* descriptors, int count, int max_rows, int max_cols, cudaStream_t stream) {
  constexpr int kCols = kTileBytes / static_cast<int>(sizeof(T));
  const dim3 grid(count, (max_rows + kRows - 1) / kRows, (max_cols + kCols - 1) / kCols);
  if (grid.y > 65535u || grid.z > 65535u) return RLT_E_LIMIT;
  return count <= kInlineSmall ? launch_inline<T, kInlineSmall>(descriptors, count, grid, stream)
                               : launch_inline<T, RLT_INLINE_TRANSFERS>(descriptors, count, grid, stream);
}

// Flat copy with conversion. A thread handles N consecutive elements, N = 32 / (size of the widest of the three types): the
// widest side moves as 32-byte accesses and the narrower sides as 16-, 8- or 4-byte ones, all of them contiguous across
// the warp. A CTA does two such groups per thread, both loaded before either is stored, and the grid holds one CTA per
// 16 KiB of the widest side, in order (block_moves.cu says why that is faster than a persistent loop). Elements before the
// first place where every pointer is aligned to its N elements, and the last few, go one at a time; tensors with no such
// place go so altogether. Bound by HBM, by L2 for what fits there. Measured, persistent kernel -> this one:
// 128 Mi elements int64 -> int32 253 -> 233 us (6.9 TB/s), float16 -> int32 143 -> 121, bfloat16 -> float16 and int64 303 -> 242;
// int32 -> int32 views that start one element past an aligned one 233 -> 159.
constexpr int kFlatGroups = 2;
// Elements per thread where nothing is aligned, all loaded before any is stored (64 Mi elements into views that start elsewhere than the source's,
// us, one by one -> so: int32 -> int32 142 -> 78, float16 -> int32 142 -> 72, bfloat16 -> float32 139 -> 68).
constexpr int kFlatSingles = 8;

template <int kBytes>
struct Bits;
template <>
struct Bits<32> { using type = Vec32; };
template <>
struct Bits<16> { using type = uint4; };
template <>
struct Bits<8> { using type = uint2; };
template <>
struct Bits<4> { using type = uint32_t; };

template <typename T, int N>
struct alignas(sizeof(T) * N) Pack {
  T v[N];
};

__device__ __forceinline__ void load_bits(const Vec32* p, Vec32* out) { *out = ld_stream(p); }
__device__ __forceinline__ void store_bits(Vec32* p, const Vec32& v) { st_stream(p, v); }
template <typename B>
__device__ __forceinline__ void load_bits(const B* p, B* out) { *out = *p; }
template <typename B>
__device__ __forceinline__ void store_bits(B* p, const B& v) { *p = v; }

template <typename T, int N>
__device__ __forceinline__ Pack<T, N> load_pack(const T* p) {
  using B = typename Bits<sizeof(T) * N>::type;
  union { B bits; Pack<T, N> pack; } u;
  load_bits(reinterpret_cast<const B*>(p), &u.bits);
  return u.pack;
}

template <typename T, int N>
__device__ __forceinline__ void store_pack(T* p, const Pack<T, N>& pack) {
  using B = typename Bits<sizeof(T) * N>::type;
  union { B bits; Pack<T, N> pack; } u;
  u.pack = pack;
  store_bits(reinterpret_cast<B*>(p), u.bits);
}

template <typename S, typename D, typename E>
constexpr int flat_width() {
  constexpr size_t pair = sizeof(S) > sizeof(D) ? sizeof(S) : sizeof(D);
  return static_cast<int>(32 / (pair > sizeof(E) ? pair : sizeof(E)));
}

template <typename S, typename D, typename E>
__device__ __forceinline__ void put_element(S v, D* dst, E* secondary, long long i) {
  dst[i] = Convert<D, S>::run(v);
  if (secondary != nullptr) secondary[i] = Convert<E, S>::run(v);
}

// head: elements before the first aligned one, -1 if there is no such place.
template <typename S, typename D, typename E>
__global__ void __launch_bounds__(kTile) flat_transfer_kernel(const S* src, D* dst, E* secondary, long long n, int head, int prefetch) {
  constexpr int N = 32 / (sizeof(S) > sizeof(D) ? (sizeof(S) > sizeof(E) ? sizeof(S) : sizeof(E))
                                                : (sizeof(D) > sizeof(E) ? sizeof(D) : sizeof(E)));
  if (prefetch && threadIdx.x == 0) {  // (further on as well: a loss where more is read than written, 172 -> 215 us for 1.2 GB int64 -> int32)
    constexpr long long kSource = static_cast<long long>(kTile) * kFlatGroups * N * sizeof(S);
    const uintptr_t from = ((reinterpret_cast<uintptr_t>(src + head) + 15) & ~uintptr_t{15}) + blockIdx.x * kSource;
    const uintptr_t end = reinterpret_cast<uintptr_t>(src + n) & ~uintptr_t{15};
    if (from < end) prefetch_l2(reinterpret_cast<const char*>(from), static_cast<int>(min(kSource, static_cast<long long>(end - from))));
  }
  follow_stream();
  if (head < 0) {
    const long long first = static_cast<long long>(blockIdx.x) * (kTile * kFlatSingles) + threadIdx.x;
    S in[kFlatSingles];
#pragma unroll
    for (int k = 0; k < kFlatSingles; ++k) {
      if (first + k * kTile < n) in[k] = src[first + k * kTile];
    }
#pragma unroll
    for (int k = 0; k < kFlatSingles; ++k) {
      if (first + k * kTile < n) put_element(in[k], dst, secondary, first + k * kTile);
    }
    return;
  }
  const long long groups = (n - head) / N;
  const long long first = static_cast<long long>(blockIdx.x) * (kTile * kFlatGroups) + threadIdx.x;
  Pack<S, N> in[kFlatGroups];
#pragma unroll
  for (int u = 0; u < kFlatGroups; ++u) {
    if (first + u * kTile < groups) in[u] = load_pack<S, N>(src + head + (first + u * kTile) * N);
  }
#pragma unroll
  for (int u = 0; u < kFlatGroups; ++u) {
    const long long g = first + u * kTile;
    if (g >= groups) continue;
    Pack<D, N> out;
#pragma unroll
    for (int k = 0; k < N; ++k) out.v[k] = Convert<D, S>::run(in[u].v[k]);
    store_pack<D, N>(dst + head + g * N, out);
    if (secondary != nullptr) {
      Pack<E, N> second;
#pragma unroll
      for (int k = 0; k < N; ++k) second.v[k] = Convert<E, S>::run(in[u].v[k]);
      store_pack<E, N>(secondary + head + g * N, second);
    }
  }
  if (blockIdx.x == 0) {  // both ends: fewer than 2 N elements
    const long long tail = head + groups * N;
    const long long i = threadIdx.x < head ? threadIdx.x : tail + (threadIdx.x - head);
    if (i < n && (i < head || i >= tail)) put_element(src[i], dst, secondary, i);
  }
}

// Elements to skip until src, dst and secondary are all aligned to `width` elements of theirs; -1 if that never happens.
int aligned_head(const void* src, size_t src_size, const void* dst, size_t dst_size, const void* secondary, size_t secondary_size,
                 int width, long long n) {
  auto aligned = [&](const void* p, size_t size, int skip) {
    return p == nullptr || (reinterpret_cast<uintptr_t>(p) + skip * size) % (size * width) == 0;
  };
  for (int skip = 0; skip < width && skip <= n; ++skip) {
    if (aligned(src, src_size, skip) && aligned(dst, dst_size, skip) && aligned(secondary, secondary_size, skip)) return skip;
  }
  return -1;
}

template <typename S, typename D>
int launch_segmented(const long long* descriptors, int count, int max_rows, int max_cols, cudaStream_t stream) {
  const dim3 grid(count, (max_rows + kRows - 1) / kRows, (max_cols + kTile - 1) / kTile);
  if (grid.y > 65535u || grid.z > 65535u) return RLT_E_LIMIT;
  RLT_CUDA_TRY(launch_following(segmented_transfer_kernel<S, D>, grid, kTile, stream, descriptors));
  return RLT_OK;
}

template <typename S, typename D, typename E>
int launch_flat_typed(const void* src, void* dst, void* secondary, long long n, cudaStream_t stream) {
  constexpr int kWidth = flat_width<S, D, E>();
  const int head = aligned_head(src, sizeof(S), dst, sizeof(D), secondary, sizeof(E), kWidth, n);
  const long long per = head < 0 ? kTile * kFlatSingles : static_cast<long long>(kTile) * kFlatGroups * kWidth;
  const long long grid = (n + per - 1) / per;
  if (grid > 0x7fffffffll) return RLT_E_LIMIT;
  const int64_t bytes = n * static_cast<int64_t>(sizeof(S) + sizeof(D) + (secondary != nullptr ? sizeof(E) : 0));
  const int prefetch = asking(head >= 0 && prefetches(src, bytes));
  RLT_CUDA_TRY(launch_following(flat_transfer_kernel<S, D, E>, static_cast<unsigned>(grid), kTile, stream, static_cast<const S*>(src),
                                static_cast<D*>(dst), static_cast<E*>(secondary), n, head, prefetch));
  return RLT_OK;
}

template <typename S, typename D>
int launch_flat(const void* src, void* dst, void* secondary, long long n, int secondary_dtype, cudaStream_t stream) {
  // no second output: its type must not narrow the vector width
  if (secondary == nullptr) return launch_flat_typed<S, D, D>(src, dst, nullptr, n, stream);
  switch (secondary_dtype) {
    case RLT_DTYPE_I32: return launch_flat_typed<S, D, int>(src, dst, secondary, n, stream);
    case RLT_DTYPE_I64: return launch_flat_typed<S, D, long long>(src, dst, secondary, n, stream);
    case RLT_DTYPE_F16: return launch_flat_typed<S, D, __half>(src, dst, secondary, n, stream);
    case RLT_DTYPE_BF16: return launch_flat_typed<S, D, __nv_bfloat16>(src, dst, secondary, n, stream);
    case RLT_DTYPE_F32: return launch_flat_typed<S, D, float>(src, dst, secondary, n, stream);
    default: return RLT_E_INVALID;
  }
}

// Calls f.template operator()<S, D>() for the pair of type codes.
template <typename F>
int dispatch_pair(int src_dtype, int dst_dtype, F f) {
#define RLT_DST(S)                                                      \
  switch (dst_dtype) {                                                  \
    case RLT_DTYPE_I32: return f.template operator()<S, int>();         \
    case RLT_DTYPE_I64: return f.template operator()<S, long long>();   \
    case RLT_DTYPE_F16: return f.template operator()<S, __half>();      \
    case RLT_DTYPE_BF16: return f.template operator()<S, __nv_bfloat16>(); \
    case RLT_DTYPE_F32: return f.template operator()<S, float>();       \
    default: return RLT_E_INVALID;                                      \
  }
  switch (src_dtype) {
    case RLT_DTYPE_I32: RLT_DST(int)
    case RLT_DTYPE_I64: RLT_DST(long long)
    case RLT_DTYPE_F16: RLT_DST(__half)
    case RLT_DTYPE_BF16: RLT_DST(__nv_bfloat16)
    case RLT_DTYPE_F32: RLT_DST(float)
    default: return RLT_E_INVALID;
  }
#undef RLT_DST
}

struct SegmentedCall {
  const long long* descriptors;
  int count, max_rows, max_cols;
  cudaStream_t stream;
  template <typename S, typename D>
  int operator()() const { return launch_segmented<S, D>(descriptors, count, max_rows, max_cols, stream); }
};

struct FlatCall {
  const void* src;
  void* dst;
  void* secondary;
  long long n;
  int secondary_dtype;
  cudaStream_t stream;
  template <typename S, typename D>
  int operator()() const { return launch_flat<S, D>(src, dst, secondary, n, secondary_dtype, stream); }
};

}  // namespace
}  // namespace rlt

extern "C" {

int rlt_tensor_transfer(const int64_t* descriptors, int32_t count, int32_t max_rows, int32_t max_cols,
                        int32_t src_dtype, int32_t dst_dtype, rlt_stream_t stream) {
  if (count == 0) return RLT_OK;
  if (descriptors == nullptr || count < 0 || max_rows < 1 || max_cols < 1) return RLT_E_INVALID;
  const rlt::SegmentedCall call{reinterpret_cast<const long long*>(descriptors), count, max_rows, max_cols,
                                reinterpret_cast<cudaStream_t>(stream)};
  const int rc = rlt::dispatch_pair(src_dtype, dst_dtype, call);
  if (rc != RLT_OK) return rc;
  RLT_CUDA_TRY(cudaGetLastError());
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

int rlt_tensor_transfer_inline(const int64_t* descriptors, int32_t count, int32_t max_rows, int32_t max_cols, int32_t dtype,
                               rlt_stream_t stream) {
  if (count == 0) return RLT_OK;
  if (descriptors == nullptr || count < 0 || max_rows < 1 || max_cols < 1) return RLT_E_INVALID;
  if (count > RLT_INLINE_TRANSFERS) return RLT_E_LIMIT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int rc = RLT_E_INVALID;
  switch (dtype) {
    case RLT_DTYPE_F16:
    case RLT_DTYPE_BF16: rc = rlt::launch_inline<uint16_t>(descriptors, count, max_rows, max_cols, s); break;
    case RLT_DTYPE_I32:
    case RLT_DTYPE_F32: rc = rlt::launch_inline<uint32_t>(descriptors, count, max_rows, max_cols, s); break;
    case RLT_DTYPE_I64: rc = rlt::launch_inline<unsigned long long>(descriptors, count, max_rows, max_cols, s); break;
  }
  if (rc != RLT_OK) return rc;
  RLT_CUDA_TRY(cudaGetLastError());
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

int rlt_tensor_copy(const void* src, void* dst, void* secondary, int64_t count, int32_t src_dtype, int32_t dst_dtype,
                    int32_t secondary_dtype, rlt_stream_t stream) {
  if (count == 0) return RLT_OK;
  if (src == nullptr || dst == nullptr || count < 0) return RLT_E_INVALID;
  const rlt::FlatCall call{src, dst, secondary, count, secondary_dtype, reinterpret_cast<cudaStream_t>(stream)};
  const int rc = rlt::dispatch_pair(src_dtype, dst_dtype, call);
  if (rc != RLT_OK) return rc;
  RLT_CUDA_TRY(cudaGetLastError());
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

}  // extern "C"
