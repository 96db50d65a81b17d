// Copies of explicit byte ranges: one range (push) or a device-resident list of
// (source, destination, bytes) triples (copy_segments).
//
// copy_segments performs the WRITE of one NixlConnector.submit call
// (vllm_rlt/pd/transport.py:182-201) for the descriptor lists that
// partition_segments produces (:95-112): up to a few hundred ranges whose sizes
// differ by orders of magnitude (a 1.5 MiB block next to a 4 KiB partial row).
//
// Work split: the ranges are cut into tiles, and the tiles of all ranges form one flat index space.
//
// Where the host knows the sizes (push, and ranges that come from the host, whose triples are kernel parameters) the grid
// holds one CTA per 16 KiB tile, in order: the hardware then keeps all SMs within a few MB of each other, which DRAM
// rewards (block_moves.cu has the measurements). 0.4 GB read and written in 256 ranges of 1.5 MiB: 136 us with the persistent kernel
// below, 120 here; a push of 1 GiB 343 -> 312 us (6.9 TB/s). Asking for the source ahead of time (prefetch_l2): 170 ranges of 1.5 MiB one
// launch behind another 81.6 -> 78.0 us, a push of 64 MiB 18.1 -> 17.5.
//
// A list in device memory has sizes the host cannot see: a persistent grid strides over tiles of 32 KiB, every CTA computes the
// exclusive scan of the per-range tile counts with warp-shuffle prefix sums in shared memory and finds a tile's range by
// binary search.
//
// Roofline: one read and one write per byte. Local copies are HBM bound; a
// destination on a peer GPU is bound by NVLink (one direction).

#include <cstring>

#include "common.cuh"
#include "internal.h"

namespace rlt {
namespace {

constexpr long long kTileBytes = 32 * 1024;   // of the persistent kernel: 16, 64 and 128 KiB, and 4 or 6 CTAs per SM, all measured slower
constexpr long long kShortTile = 16 * 1024;   // of one CTA per tile
constexpr int kCtasPerSm = 3;

// Asks for the source of a tile, but for the bytes at its ends that share 16 with others.
__device__ __forceinline__ void prefetch_tile(const char* src, long long n) {
  const int skip = static_cast<int>(-reinterpret_cast<intptr_t>(src) & 15);
  if (n >= skip + 16) prefetch_l2(src + skip, static_cast<int>(n - skip) & ~15);
}

__global__ void __launch_bounds__(kThreads, 6) push_kernel(const char* src, char* dst, long long nbytes, int prefetch) {
  const long long at = static_cast<long long>(blockIdx.x) * kShortTile;
  if (prefetch && threadIdx.x < 2) {
    const long long from = at + (threadIdx.x ? kPrefetchAhead * kShortTile : 0);
    if (from < nbytes) prefetch_tile(src + from, min(kShortTile, nbytes - from));
  }
  follow_stream();
  copy_piece<true>(src + at, dst + at, min(kShortTile, nbytes - at));
}

struct Segment {
  const char* src;
  char* dst;
  long long bytes;
};
template <int kCount>
struct InlineSegments {
  int count;
  int prefetch;
  int first_tile[kCount + 1];
  Segment segment[kCount];
};

template <int kCount>
__global__ void __launch_bounds__(kThreads, 6) inline_segments_kernel(const __grid_constant__ InlineSegments<kCount> list) {
  struct Tile {
    const char* src;
    char* dst;
    long long bytes;
  };
  const auto tile_at = [&](int t) -> Tile {
    int lo = 0, hi = list.count;  // last range whose first tile is at or before t
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (list.first_tile[mid] <= t) lo = mid; else hi = mid;
    }
    const Segment& s = list.segment[lo];
    const long long at = static_cast<long long>(t - list.first_tile[lo]) * kShortTile;
    return {s.src + at, s.dst + at, min(kShortTile, s.bytes - at)};
  };
  const Tile tile = tile_at(static_cast<int>(blockIdx.x));
  if (list.prefetch) {
    if (threadIdx.x == 0) prefetch_tile(tile.src, tile.bytes);
    if (threadIdx.x == 32 && gridDim.x - blockIdx.x > kPrefetchAhead) {
      const Tile next = tile_at(static_cast<int>(blockIdx.x + kPrefetchAhead));
      prefetch_tile(next.src, next.bytes);
    }
  }
  follow_stream();
  copy_piece<true>(tile.src, tile.dst, tile.bytes);
}

template <int kCount>
int launch_inline(const int64_t* triples, int count, cudaStream_t stream) {
  InlineSegments<kCount> list;
  long long tiles = 0, bytes = 0;
  list.count = 0;
  for (int i = 0; i < count; ++i) {
    if (triples[3 * i + 2] <= 0) continue;
    list.first_tile[list.count] = static_cast<int>(tiles);
    list.segment[list.count++] = {reinterpret_cast<const char*>(triples[3 * i]), reinterpret_cast<char*>(triples[3 * i + 1]), triples[3 * i + 2]};
    tiles += (triples[3 * i + 2] + kShortTile - 1) / kShortTile;
    bytes += triples[3 * i + 2];
    if (tiles > 0x7fffffffll) return RLT_E_LIMIT;
  }
  if (list.count == 0) return RLT_OK;
  list.first_tile[list.count] = static_cast<int>(tiles);
  // Every range has to be in this GPU's memory: a list may take them from anywhere. (All of a worker's pools: one look-up a tensor.)
  bool ask = 2 * bytes >= kPrefetchBytes;
  OwnMemory mine;
  for (int i = 0; ask && i < list.count; ++i) ask = mine.holds(list.segment[i].src, list.segment[i].bytes);
  list.prefetch = asking(ask);
  RLT_CUDA_TRY(launch_following(inline_segments_kernel<kCount>, static_cast<unsigned>(tiles), kThreads, stream, list));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

__global__ void __launch_bounds__(kThreads, 3) segment_copy_kernel(const long long* __restrict__ segments, int count) {
  extern __shared__ int tile_off[];  // [count + 1] exclusive scan of tiles per range
  __shared__ int warp_sum[kThreads / 32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    carry = 0;
    tile_off[0] = 0;
  }
  __syncthreads();
  for (int base = 0; base < count; base += kThreads) {
    const int s = base + threadIdx.x;
    int tiles = 0;
    if (s < count) {
      const long long n = segments[3ll * s + 2];
      tiles = n > 0 ? static_cast<int>((n + kTileBytes - 1) / kTileBytes) : 0;
    }
    const int inc = warp_inclusive_scan(tiles);
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; ++w) before += warp_sum[w];
    if (s < count) tile_off[s + 1] = before + inc;
    __syncthreads();
    if (threadIdx.x == kThreads - 1) carry = before + inc;
    __syncthreads();
  }
  const int total = tile_off[count];
  for (int t = blockIdx.x; t < total; t += gridDim.x) {
    int lo = 0, hi = count;  // last range whose first tile is at or before t
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile_off[mid] <= t) lo = mid; else hi = mid;
    }
    const long long at = static_cast<long long>(t - tile_off[lo]) * kTileBytes;
    const long long n = segments[3ll * lo + 2];
    copy_piece<false>(reinterpret_cast<const char*>(segments[3ll * lo]) + at, reinterpret_cast<char*>(segments[3ll * lo + 1]) + at,
               min(kTileBytes, n - at));
  }
}

}  // namespace
}  // namespace rlt

extern "C" {

int rlt_kv_push(const void* src, void* dst, int64_t nbytes, rlt_stream_t stream) {
  const rlt::NvtxRange range("rlt.kv_push");
  if (nbytes == 0) return RLT_OK;
  if (src == nullptr || dst == nullptr || nbytes < 0) return RLT_E_INVALID;
  const long long tiles = (nbytes + rlt::kShortTile - 1) / rlt::kShortTile;
  if (tiles > 0x7fffffffll) return RLT_E_LIMIT;
  RLT_CUDA_TRY(rlt::launch_following(rlt::push_kernel, static_cast<unsigned>(tiles), rlt::kThreads, reinterpret_cast<cudaStream_t>(stream),
                                     static_cast<const char*>(src), static_cast<char*>(dst), static_cast<long long>(nbytes),
                                     static_cast<int>(rlt::asking(rlt::prefetches(src, 2 * nbytes)))));
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

int rlt_copy_segments_inline(const int64_t* triples, int32_t count, rlt_stream_t stream) {
  const rlt::NvtxRange range("rlt.kv_copy_segments");
  if (count == 0) return RLT_OK;
  if (triples == nullptr || count < 0) return RLT_E_INVALID;
  if (count > RLT_INLINE_SEGMENTS) return RLT_E_LIMIT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // a parameter block is copied into the launch whole: 256 ranges are what one submission of the default configuration holds
  return count <= 32    ? rlt::launch_inline<32>(triples, count, s)
         : count <= 256 ? rlt::launch_inline<256>(triples, count, s)
                        : rlt::launch_inline<RLT_INLINE_SEGMENTS>(triples, count, s);
}

int rlt_load_segments(void) {
  using namespace rlt;
  RLT_CUDA_TRY(load_kernel(push_kernel));
  RLT_CUDA_TRY(load_kernel(inline_segments_kernel<32>));
  RLT_CUDA_TRY(load_kernel(inline_segments_kernel<256>));
  RLT_CUDA_TRY(load_kernel(inline_segments_kernel<RLT_INLINE_SEGMENTS>));
  return RLT_OK;
}

int rlt_kv_copy_segments(const int64_t* segments, int32_t count, rlt_stream_t stream) {
  const rlt::NvtxRange range("rlt.kv_copy_segments");
  if (count == 0) return RLT_OK;
  if (segments == nullptr || count < 0) return RLT_E_INVALID;
  if (count > RLT_MAX_SEGMENTS) return RLT_E_LIMIT;
  int sms = 0;
  const int rc = rlt::sm_count(&sms);
  if (rc != RLT_OK) return rc;
  const size_t smem = (static_cast<size_t>(count) + 1) * sizeof(int);
  rlt::segment_copy_kernel<<<sms * rlt::kCtasPerSm, rlt::kThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const long long*>(segments), count);
  RLT_CUDA_TRY(cudaGetLastError());
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

}  // extern "C"
