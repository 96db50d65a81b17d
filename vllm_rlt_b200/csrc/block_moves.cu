// Handoff, pack and scatter from per-page records (block_moves.h): the kernels of a batch whose tables the host holds.
//
// Work decomposition. Inside a KV block the rows lie [layer][token][row], so a layer slice of a block is one contiguous
// byte range on every plane of either pool. A CTA takes one small piece of such a range, 8 or 16 KiB, of one page:
// vector i of the piece sits at the same offset of the source and of the destination block, and which token it belongs
// to matters only where a page is partly in range, where exit planes choose the source, or where a packed image is
// compacted. There is no loop over units: the grid holds one CTA per piece, in address order.
//
// Why small pieces and no persistent loop: the memory system is fastest when the bytes in flight at any moment are
// neighbours. The hardware hands pieces to SMs in order as they become free, which keeps all SMs within a few MB of each
// other; CTAs that stride over the work drift apart. Measured on one B200 with 1 GiB per stream, against 444
// persistent CTAs: one read per write 6.2 -> 6.9 TB/s, one read per two writes 5.7 -> 6.85, per three 5.65 -> 6.8, per seven
// 5.4 -> 6.7 (pieces of 8 KiB; 16 KiB within 1 %, 64 KiB 4 % slower), of which 32-byte accesses are 1 - 3 %.
//
// What a CTA must know is read in one round from the page's record; for small batches the records are kernel parameters, so a
// launch needs no staging copy before it. Block ids and exit planes are checked here and reported in the status words;
// a row that fails is skipped.

#include <algorithm>
#include <cstring>

#include "block_moves.h"
#include "common.cuh"
#include "table_params.cuh"

namespace rlt {
namespace {

enum MoveKind {
  kPlaneToPlane,   // ALL_PLANES handoff: plane p <- plane p
  kExitToPlane,    // EXIT_ONLY handoff: the only plane <- the token's exit plane
  kFanOut,         // DEDUP handoff: planes up to the exit plane are read once, deeper ones filled from the last
  kPlaneToWire,    // pack, ALL_PLANES
  kExitToWire,     // pack, EXIT_ONLY
  kDedupToWire,    // pack, DEDUP
  kWireToPlane,    // scatter of an image with every plane
  kDedupFromWire,  // scatter of a dedup image: like kFanOut with the rows taken from the image
  // the same two with images whose rows are at odd places (load_image): kernels of their own, because the registers of that would cost the
  // others 1 - 5 %
  kDedupToOddWire,
  kDedupFromOddWire
};

__host__ __device__ constexpr bool by_token(MoveKind k) { return k == kExitToPlane || k == kExitToWire; }
__host__ __device__ constexpr bool asks_ahead(MoveKind k) { return k == kPlaneToPlane || k == kPlaneToWire || k == kWireToPlane || by_token(k); }
__host__ __device__ constexpr bool packs_dedup(MoveKind k) { return k == kDedupToWire || k == kDedupToOddWire; }
__host__ __device__ constexpr bool scatters_dedup(MoveKind k) { return k == kDedupFromWire || k == kDedupFromOddWire; }
__host__ __device__ constexpr bool loops_planes(MoveKind k) { return k == kFanOut || scatters_dedup(k); }

struct MoveRegion {
  const char* src[2];  // K and V; the image for a scatter
  char* dst[2];
  long long block_bytes;
  long long slice_at;  // byte offset of the layer slice inside a block
  int token_bytes;
  int vec_bytes;       // 32, 16, 4 or 1: what the pools' rows allow
  int image_bytes;     // 16, 8 or 4: of one access to the image where the vectors have 16
  int row_vecs;
  unsigned row_magic;  // div_magic(row_vecs), 0 for one-vector rows
  int slice_vecs;      // vectors of the layer slice of one block
  int pieces;          // CTAs per (page, plane, K|V)
  int per;             // vectors of one piece
};

struct MoveParams {
  MoveRegion region[2];
  int pieces;        // CTAs per (page, plane of the grid): 2 * (region[0].pieces + region[1].pieces)
  int grid_planes;   // planes the grid enumerates (1 where a CTA walks the planes itself)
  int plane_begin, plane_end;
  int src_planes, dst_planes, src_blocks, dst_blocks;
  int block_size;
  unsigned block_magic;
  int layer_begin, slice_layers;
  unsigned long long deep_layer_mask;
  long long packed_bytes, packed_token_bytes;
  int words;         // int32 per record
  int blocks;
  int dst_at, exit_at;  // where a record's destination blocks and exit planes start
  const int* records;
  const int* wire;   // [blocks][planes]
  long long* wire_header;
  long long wire_tokens;
  int* status;
};

template <int kWords>
struct MoveArgs {
  MoveParams p;
  int inline_words[kWords];
};

// Vectors per thread of one piece, and how many of them are in flight together: 16 KiB pieces where a vector is read
// and written once, 8 KiB per plane where the planes are walked (their loads are batched over planes instead). Narrow
// vectors get smaller pieces.
template <typename T>
__host__ __device__ constexpr int unroll_of(bool planes) {
  return sizeof(T) == 32 ? (planes ? 1 : 2) : sizeof(T) == 16 ? (planes ? 2 : 4) : sizeof(T) == 4 ? 8 : 16;
}
template <typename T>
__host__ __device__ constexpr int flight_of() {
  return sizeof(T) == 32 ? 2 : 4;
}

struct Piece {
  const int* rec;
  int g, kv, index, plane;
  int t_lo, t_hi;
  // read again where an error is reported, not kept in registers for it
  __device__ int request() const { return rec[0]; }
  __device__ int logical() const { return rec[1]; }
};

// A page's record as the kinds that choose planes per token use it: fetched by the CTA in one round, then looked up in
// shared memory (a chain of global lookups, token -> exit plane -> block, would cost a CTA this short as much time as its
// payload).
constexpr int kMaxPlanes = kMaxRecordPlanes;
struct PageShared {
  long long src[kMaxPlanes];  // byte offset of each plane's block, -1 if the id is outside the pool
  long long dst[kMaxPlanes];
  long long wire[kMaxPlanes];               // dedup image: where this page's rows of each plane start
  unsigned long long carried[kMaxPlanes];   // dedup image: tokens of the page that the plane carries
  int src_id[kMaxPlanes], dst_id[kMaxPlanes];
  int exit_plane[kMaxBlockSize];
};
// kDedupToWire: the (token, plane) pairs of a page that are on the wire, token by token (plane << 8 | token).
struct PagePairs {
  unsigned short code[kMaxPlanes * kMaxBlockSize];
};

// Where vector `k` behind the piece's first one is: row (layer-major, token-minor), token, and vector inside the row. The piece's rows are those of
// `tokens` tokens from `t_lo` on, layer by layer: a whole block's, or only the ones in range. k counts from the piece's first vector, whose row and
// offset are (row0, rem0): the multiplier split stays exact.
struct RowAt {
  int layer, token, within;
};
__device__ __forceinline__ RowAt row_at(const MoveRegion& rg, int tokens, unsigned magic, int t_lo, int row0, int rem0, int k) {
  const unsigned j = static_cast<unsigned>(rem0 + k);
  const int q = rg.row_magic ? static_cast<int>(__umulhi(j, rg.row_magic)) : static_cast<int>(j);
  const int row = row0 + q;
  const int layer = tokens == 1 ? row : static_cast<int>(__umulhi(static_cast<unsigned>(row), magic));
  return {layer, t_lo + row - layer * tokens, static_cast<int>(j) - q * rg.row_vecs};
}

// A vector of the image; kSplit: in pieces of 8 or 4 bytes, because its rows follow one another whatever their size. (FP8 codes beside the scales
// of an odd number of heads lie on 4-byte boundaries in the image and on 16-byte ones in the pool. Where a row is found by arithmetic, doing that for
// 16 bytes and not for 4 halves the time: 15 prompts of 7 planes and 384-byte rows, dedup, packed in 309 us instead of 660 and scattered in 419
// instead of 783; 56 prompts with every plane scattered in 470 instead of 708.)
template <bool kSplit, typename T>
__device__ __forceinline__ T load_image(const char* from, int bytes) {
  if constexpr (!kSplit) {
    return ld_stream(reinterpret_cast<const T*>(from));
  } else {
    static_assert(sizeof(T) == 16, "");
    const uint32_t* w = reinterpret_cast<const uint32_t*>(from);
    if (bytes == 4) return T{w[0], w[1], w[2], w[3]};
    const uint2 lo = *reinterpret_cast<const uint2*>(from), hi = *reinterpret_cast<const uint2*>(from + 8);
    return T{lo.x, lo.y, hi.x, hi.y};
  }
}
template <bool kSplit, typename T>
__device__ __forceinline__ void store_image(char* to, const T& v, int bytes) {
  if constexpr (!kSplit) {
    st_stream(reinterpret_cast<T*>(to), v);
  } else {
    static_assert(sizeof(T) == 16, "");
    uint32_t* w = reinterpret_cast<uint32_t*>(to);
    if (bytes == 4) {
      w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else {
      *reinterpret_cast<uint2*>(to) = uint2{v.x, v.y};
      *reinterpret_cast<uint2*>(to + 8) = uint2{v.z, v.w};
    }
  }
}

// `count` vectors of 16 bytes to a place in the image that is only a multiple of 4: the image's vectors are stored whole, and each is put together
// from four words of the source, which lie in L1 by the second of them: 56 prompts with every plane packed in 454 us, 713 with 4-byte accesses on both
// sides, 1,430 with the source's vectors stored in four parts each.
__device__ __forceinline__ void copy_to_odd_place(const char* from, char* to, int count) {
  const int skip = static_cast<int>(-reinterpret_cast<intptr_t>(to) & 15);
  const int words = count * 4, head = skip / 4, body = (words - head) / 4, done = head + 4 * body;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(from);
  constexpr int kU = 4;
  for (int k0 = static_cast<int>(threadIdx.x); k0 < body; k0 += kThreads * kU) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t* w = src + head + 4 * (k0 + u * kThreads);
      if (k0 + u * kThreads < body) v[u] = uint4{w[0], w[1], w[2], w[3]};
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (k0 + u * kThreads < body) st_stream(reinterpret_cast<uint4*>(to + skip) + k0 + u * kThreads, v[u]);
    }
  }
  const int i = static_cast<int>(threadIdx.x);
  uint32_t* dst = reinterpret_cast<uint32_t*>(to);
  if (i < head) dst[i] = src[i];
  if (i < words - done) dst[done + i] = src[done + i];
}

__device__ __forceinline__ bool deep_carried(const MoveParams& p, int layer_rel) {
  return p.deep_layer_mask == 0 || ((p.deep_layer_mask >> (p.layer_begin + layer_rel)) & 1ull) != 0;
}

// The block's address offset, or -1 (reported) if its id is outside the pool.
__device__ __forceinline__ long long block_at(const MoveParams& p, const MoveRegion& rg, const Piece& w, int id, int blocks) {
  if (static_cast<unsigned>(id) < static_cast<unsigned>(blocks)) return id * rg.block_bytes;
  report(p.status, RLT_STATUS_BAD_BLOCK, w.request(), w.logical(), id);
  return -1;
}

// The same from the page's shared table.
__device__ __forceinline__ long long used_block(const MoveParams& p, const Piece& w, long long offset, int id) {
  if (offset < 0) report(p.status, RLT_STATUS_BAD_BLOCK, w.request(), w.logical(), id);
  return offset;
}

// Offset in the image of the first row of (page, plane, region, K|V) when `tokens` of the page are carried there.
__device__ __forceinline__ long long wire_base(const MoveParams& p, const Piece& w, const MoveRegion& rg, long long before,
                                               int tokens) {
  long long at = before * p.packed_token_bytes;
  if (w.g == 1) at += 2ll * p.slice_layers * tokens * p.region[0].token_bytes;
  return at + static_cast<long long>(w.kv) * p.slice_layers * tokens * rg.token_bytes;
}

template <MoveKind K>
__device__ __forceinline__ void fetch_page(const MoveParams& p, const MoveRegion& rg, const Piece& w, const int* wire, PageShared& s) {
  constexpr bool kImage = packs_dedup(K) || scatters_dedup(K);
  const int tid = static_cast<int>(threadIdx.x);
  const int word = kRecordHeader + tid;
  if (word < p.words) {
    const int v = w.rec[word];
    if (word >= p.exit_at) {
      s.exit_plane[word - p.exit_at] = v;
    } else if (word >= p.dst_at) {
      s.dst_id[word - p.dst_at] = v;
      s.dst[word - p.dst_at] = static_cast<unsigned>(v) < static_cast<unsigned>(p.dst_blocks) ? v * rg.block_bytes : -1;
    } else {
      s.src_id[tid] = v;
      s.src[tid] = static_cast<unsigned>(v) < static_cast<unsigned>(p.src_blocks) ? v * rg.block_bytes : -1;
    }
  }
  long long before = 0;
  const int planes = p.src_planes;
  const int lane = tid & 31, warp = tid >> 5;
  // warp w looks after planes w, w + 8, ...; its lane k keeps the wire entry of the k-th of them
  if (kImage && warp + lane * (kThreads / 32) < planes) before = wire[warp + lane * (kThreads / 32)];
  __syncthreads();
  if constexpr (kImage) {
    const int e0 = lane >= w.t_lo && lane < w.t_hi ? s.exit_plane[lane] : -1;
    const int e1 = lane + 32 >= w.t_lo && lane + 32 < w.t_hi ? s.exit_plane[lane + 32] : -1;
    for (int k = 0, plane = warp; plane < planes; ++k, plane += kThreads / 32) {
      const unsigned long long mask = static_cast<unsigned long long>(__ballot_sync(0xffffffffu, e0 >= plane)) |
                                      static_cast<unsigned long long>(__ballot_sync(0xffffffffu, e1 >= plane)) << 32;
      const long long first = __shfl_sync(0xffffffffu, before, k);
      if (lane == 0) {
        s.carried[plane] = mask;
        s.wire[plane] = wire_base(p, w, rg, first, __popcll(mask));
      }
    }
    __syncthreads();
  }
}

template <typename T, MoveKind K, bool kSplit>
__device__ __forceinline__ void move_rows(const MoveParams& p, const MoveRegion& rg, const Piece& w, const PageShared& s) {
  constexpr int kU = flight_of<T>();
  constexpr bool kFromImage = K == kWireToPlane, kToImage = K == kPlaneToWire || K == kExitToWire;
  const int first = w.index * rg.per;
  const int n_tok = w.t_hi - w.t_lo;
  const int sid = K == kWireToPlane || K == kExitToPlane || K == kExitToWire ? 0 : w.rec[kRecordHeader + w.plane];
  const int did = K == kPlaneToWire || K == kExitToWire ? 0 : w.rec[p.dst_at + w.plane];
  const char* src = rg.src[w.kv];
  char* dst = rg.dst[w.kv];
  long long image = 0;  // where the page's rows start in the image
  if (K == kPlaneToWire || K == kExitToWire || K == kWireToPlane) {
    const long long before = static_cast<long long>(w.rec[4]) * p.dst_planes + static_cast<long long>(w.plane) * w.rec[5] + w.rec[3];
    image = wire_base(p, w, rg, before, n_tok);
  }
  if (K == kPlaneToPlane || K == kPlaneToWire) {
    const long long at = block_at(p, rg, w, sid, p.src_blocks);
    if (at < 0) return;
    src += at + rg.slice_at;
  } else if (K == kWireToPlane) {
    src += image;
  }
  if (K == kPlaneToPlane || K == kExitToPlane || K == kWireToPlane) {
    const long long at = block_at(p, rg, w, did, p.dst_blocks);
    if (at < 0) return;
    dst += at + rg.slice_at;
  } else {
    dst += image;
  }
  T regs[kU];
  // A page that is carried whole is the same byte range on both sides, the image included.
  const bool whole = n_tok == p.block_size && (w.plane == 0 || p.deep_layer_mask == 0) &&
                     (K == kPlaneToPlane || K == kExitToPlane ||
                      image + static_cast<long long>(rg.slice_vecs) * static_cast<int>(sizeof(T)) <= p.packed_bytes);
  if (K != kExitToPlane && K != kExitToWire && whole) {
    const T* from = reinterpret_cast<const T*>(src) + first;
    T* to = reinterpret_cast<T*>(dst) + first;
    const int left = rg.slice_vecs - first;
    if (kSplit && kToImage) {
      if (left > 0) copy_to_odd_place(reinterpret_cast<const char*>(from), reinterpret_cast<char*>(to), min(left, rg.per));
      return;
    }
    for (int k0 = static_cast<int>(threadIdx.x); k0 < rg.per; k0 += kThreads * kU) {
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if (k0 + u * kThreads < left) regs[u] = kFromImage ? load_image<kSplit, T>(reinterpret_cast<const char*>(from + k0 + u * kThreads), rg.image_bytes) : ld_stream(from + k0 + u * kThreads);
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if (k0 + u * kThreads >= left) continue;
        if (kToImage) store_image<kSplit>(reinterpret_cast<char*>(to + k0 + u * kThreads), regs[u], rg.image_bytes);
        else st_stream(to + k0 + u * kThreads, regs[u]);
      }
    }
    return;
  }
  const int row0 = first / rg.row_vecs, rem0 = first - row0 * rg.row_vecs;
  for (int k0 = static_cast<int>(threadIdx.x); k0 < rg.per; k0 += kThreads * kU) {
    char* to[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int k = k0 + u * kThreads;
      to[u] = nullptr;
      if (first + k >= rg.slice_vecs) continue;
      const RowAt at = row_at(rg, p.block_size, p.block_magic, 0, row0, rem0, k);
      if (at.token < w.t_lo || at.token >= w.t_hi) continue;
      if (w.plane > 0 && !deep_carried(p, at.layer)) continue;
      const long long in_slice = static_cast<long long>(first + k) * static_cast<int>(sizeof(T));
      long long in_image = 0;
      if (K == kPlaneToWire || K == kExitToWire || K == kWireToPlane) {
        in_image = (static_cast<long long>(at.layer) * n_tok + (at.token - w.t_lo)) * rg.token_bytes;
        if (image + in_image + rg.token_bytes > p.packed_bytes) {
          report(p.status, RLT_STATUS_BAD_RANGE, w.request(), w.logical() * p.block_size + w.t_lo, w.logical() * p.block_size + w.t_hi);
          continue;
        }
        in_image += static_cast<long long>(at.within) * static_cast<int>(sizeof(T));
      }
      const char* from = src + (K == kWireToPlane ? in_image : in_slice);
      if (K == kExitToPlane || K == kExitToWire) {
        const int e = s.exit_plane[at.token];
        if (e < 0 || e >= p.src_planes) {
          report(p.status, RLT_STATUS_BAD_PLANE, w.request(), w.logical() * p.block_size + at.token, e);
          continue;
        }
        const long long block = used_block(p, w, s.src[e], s.src_id[e]);
        if (block < 0) continue;
        from += block + rg.slice_at;
      }
      to[u] = dst + (kToImage ? in_image : in_slice);
      regs[u] = kFromImage ? load_image<kSplit, T>(from, rg.image_bytes) : ld_stream(reinterpret_cast<const T*>(from));
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (to[u] == nullptr) continue;
      if (kToImage) store_image<kSplit>(to[u], regs[u], rg.image_bytes);
      else st_stream(reinterpret_cast<T*>(to[u]), regs[u]);
    }
  }
}

// The kinds that walk the planes: every row of planes up to the token's exit plane is read once; the last one is also
// what the deeper planes get (kFanOut, kDedupFromWire). kPlaneBatch loads of a thread are in flight before the
// first store.
constexpr int kPlaneBatch = 4;

template <typename T, MoveKind K, bool kSplit>
__device__ __forceinline__ void walk_planes(const MoveParams& p, const MoveRegion& rg, const Piece& w, const PageShared& s) {
  const int first = w.index * rg.per;
  const int row0 = first / rg.row_vecs, rem0 = first - row0 * rg.row_vecs;
  const int begin = p.plane_begin;
  // A handoff goes through the rows in range only, a scatter through the block's: us of the one and the other, handoffs of 5 GB and two planes
  // 854 / 872, of 480-byte rows 808 / 833, scatters of 5 GB and two planes 909 / 902, of a hundred pages 105 / 103.
  constexpr bool kInRange = K == kFanOut;
  const int tokens = kInRange ? w.t_hi - w.t_lo : p.block_size, t_lo = kInRange ? w.t_lo : 0;
  const unsigned magic = !kInRange || tokens == p.block_size || tokens == 1 ? p.block_magic : 0xffffffffu / static_cast<unsigned>(tokens) + 1u;
  const int count = min(rg.per, (kInRange ? p.slice_layers * tokens * rg.row_vecs : rg.slice_vecs) - first);
  for (int k = static_cast<int>(threadIdx.x); k < count; k += kThreads) {
    const RowAt at = row_at(rg, tokens, magic, t_lo, row0, rem0, k);
    if (!kInRange && (at.token < w.t_lo || at.token >= w.t_hi)) continue;
    const int e = s.exit_plane[at.token];
    if (e < 0 || e >= p.src_planes) {
      report(p.status, RLT_STATUS_BAD_PLANE, w.request(), w.logical() * p.block_size + at.token, e);
      continue;
    }
    const char* src = rg.src[w.kv];
    char* dst = rg.dst[w.kv];
    const int vec = kInRange ? (at.layer * p.block_size + at.token) * rg.row_vecs + at.within : first + k;
    const long long in_slice = rg.slice_at + static_cast<long long>(vec) * static_cast<int>(sizeof(T));
    const int end = p.plane_end > 1 && !deep_carried(p, at.layer) ? 1 : p.plane_end;  // planes this row reaches
    if (begin >= end) continue;
    // source rows are those of planes [begin, begin + loads): plane p <- min(p, e)
    const int loads = max(1, min(e + 1, end) - begin);
    const int within = at.within * static_cast<int>(sizeof(T));
    const unsigned long long below = (1ull << at.token) - 1ull;
    // this row's offset in the image for one of the planes that carry it, -1 (reported) past the image's end
    auto image_at = [&](int plane) -> long long {
      const unsigned long long mask = s.carried[plane];
      const long long row = s.wire[plane] + (static_cast<long long>(at.layer) * __popcll(mask) + __popcll(mask & below)) * rg.token_bytes;
      if (row + rg.token_bytes <= p.packed_bytes) return row + within;
      report(p.status, RLT_STATUS_BAD_RANGE, w.request(), w.logical() * p.block_size + w.t_lo, w.logical() * p.block_size + w.t_hi);
      return -1;
    };
    T last;
    bool last_ok = false;
    for (int j0 = 0; j0 < loads; j0 += kPlaneBatch) {
      T regs[kPlaneBatch];
      bool ok[kPlaneBatch];
#pragma unroll
      for (int j = 0; j < kPlaneBatch; ++j) {
        const int plane = begin + j0 + j;
        ok[j] = j0 + j < loads;
        if (!ok[j]) continue;
        long long from;
        if (scatters_dedup(K)) {
          from = image_at(plane);
          ok[j] = from >= 0;
        } else {
          const int sp = min(plane, e);
          from = used_block(p, w, s.src[sp], s.src_id[sp]);
          ok[j] = from >= 0;
          from += in_slice;
        }
        if (ok[j]) regs[j] = scatters_dedup(K) ? load_image<kSplit, T>(src + from, rg.image_bytes) : ld_stream(reinterpret_cast<const T*>(src + from));
      }
#pragma unroll
      for (int j = 0; j < kPlaneBatch; ++j) {
        const int plane = begin + j0 + j;
        if (j0 + j >= loads) continue;
        const long long to = used_block(p, w, s.dst[plane], s.dst_id[plane]);
        if (ok[j] && to >= 0) st_stream(reinterpret_cast<T*>(dst + to + in_slice), regs[j]);
        last_ok = ok[j];
        if (ok[j]) last = regs[j];
      }
    }
    if (last_ok) {
      for (int plane = begin + loads; plane < end; ++plane) {
        const long long to = used_block(p, w, s.dst[plane], s.dst_id[plane]);
        if (to >= 0) st_stream(reinterpret_cast<T*>(dst + to + in_slice), last);
      }
    }
  }
}

// Lists the pairs of the page; returns how many. Every warp scans the tokens' plane counts for itself.
__device__ __forceinline__ int list_pairs(const MoveParams& p, const Piece& w, const PageShared& s, PagePairs& pairs) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int start[2], total = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = lane + 32 * h;
    int planes = 0;
    if (t >= w.t_lo && t < w.t_hi) {
      const int e = s.exit_plane[t];
      planes = e < 0 ? 0 : min(e + 1, p.src_planes);
    }
    const int through = warp_inclusive_scan(planes);
    start[h] = total + through - planes;
    total += __shfl_sync(0xffffffffu, through, 31);
  }
  for (int t = warp; t < p.block_size; t += kThreads / 32) {
    const int from = __shfl_sync(0xffffffffu, t < 32 ? start[0] : start[1], t & 31);
    if (t < w.t_lo || t >= w.t_hi) continue;
    const int planes = min(s.exit_plane[t] + 1, p.src_planes);
    for (int plane = lane; plane < planes; plane += 32) pairs.code[from + plane] = static_cast<unsigned short>(plane << 8 | t);
  }
  __syncthreads();
  return total;
}

// Dedup pack. What a page contributes differs from page to page, so its vectors - (layer, pair, vector of the row) - are
// dealt to the page's CTAs in equal shares: every thread has something to copy, whatever the exit planes.
template <typename T, bool kSplit>
__device__ __forceinline__ void pack_pairs(const MoveParams& p, const MoveRegion& rg, const Piece& w, const PageShared& s,
                                           PagePairs& pairs) {
  constexpr int kU = flight_of<T>();
  const int n = list_pairs(p, w, s, pairs);
  if (w.index == 0 && w.g == 0 && w.kv == 0) {  // one CTA of the page looks for tokens whose exit plane is no plane
    const int t = static_cast<int>(threadIdx.x);
    if (t >= w.t_lo && t < w.t_hi && (s.exit_plane[t] < 0 || s.exit_plane[t] >= p.src_planes))
      report(p.status, RLT_STATUS_BAD_PLANE, w.request(), w.logical() * p.block_size + t, s.exit_plane[t]);
  }
  if (n == 0) return;
  const unsigned n_magic = n == 1 ? 0u : static_cast<unsigned>((1ull << 32) / static_cast<unsigned>(n)) + 1u;
  const long long all = static_cast<long long>(p.slice_layers) * n * rg.row_vecs;
  const int first = static_cast<int>(all * w.index / rg.pieces);
  const int count = static_cast<int>(all * (w.index + 1) / rg.pieces) - first;
  const int row0 = first / rg.row_vecs, rem0 = first - row0 * rg.row_vecs;
  const char* src = rg.src[w.kv] + rg.slice_at;
  char* dst = rg.dst[w.kv];
  for (int k0 = static_cast<int>(threadIdx.x); k0 < count; k0 += kThreads * kU) {
    T regs[kU];
    char* to[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int k = k0 + u * kThreads;
      to[u] = nullptr;
      if (k >= count) continue;
      const unsigned j = static_cast<unsigned>(rem0 + k);
      const int q = rg.row_magic ? static_cast<int>(__umulhi(j, rg.row_magic)) : static_cast<int>(j);
      const int row = row0 + q;
      const int layer = n_magic ? static_cast<int>(__umulhi(static_cast<unsigned>(row), n_magic)) : row;
      const int code = pairs.code[row - layer * n];
      const int plane = code >> 8, token = code & 0xff;
      if (s.exit_plane[token] >= p.src_planes) continue;  // reported above
      const unsigned long long mask = s.carried[plane];
      const long long image = s.wire[plane] + (static_cast<long long>(layer) * __popcll(mask) + __popcll(mask & ((1ull << token) - 1ull))) * rg.token_bytes;
      if (image + rg.token_bytes > p.packed_bytes) {
        report(p.status, RLT_STATUS_BAD_RANGE, w.request(), w.logical() * p.block_size + w.t_lo, w.logical() * p.block_size + w.t_hi);
        continue;
      }
      const long long block = used_block(p, w, s.src[plane], s.src_id[plane]);
      if (block < 0) continue;
      const int within = (static_cast<int>(j) - q * rg.row_vecs) * static_cast<int>(sizeof(T));
      regs[u] = ld_stream(reinterpret_cast<const T*>(src + block + (static_cast<long long>(layer) * p.block_size + token) * rg.token_bytes + within));
      to[u] = dst + image + within;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (to[u] != nullptr) store_image<kSplit>(to[u], regs[u], rg.image_bytes);
    }
  }
}

// Which piece CTA `at` of the grid takes.
__device__ __forceinline__ Piece piece_at(const MoveParams& p, const int* records, unsigned at) {
  Piece w;
  const unsigned page = at / (static_cast<unsigned>(p.pieces) * p.grid_planes);
  at -= page * (static_cast<unsigned>(p.pieces) * p.grid_planes);
  const unsigned plane = at / p.pieces;
  at -= plane * p.pieces;
  w.plane = p.plane_begin + static_cast<int>(plane);
  w.g = at >= 2u * p.region[0].pieces;
  if (w.g) at -= 2u * p.region[0].pieces;
  const int pieces = p.region[w.g].pieces;
  w.kv = at >= static_cast<unsigned>(pieces);
  w.index = static_cast<int>(at) - w.kv * pieces;
  w.rec = records + static_cast<long long>(page) * p.words;
  return w;
}

// A warp asks for the source of a piece of a page that is wholly in range, or for the rows that its tokens' exit planes choose. Nothing is read
// but the record.
template <MoveKind K>
__device__ __forceinline__ void prefetch_piece(const MoveParams& p, const Piece& w) {
  const MoveRegion& rg = p.region[w.g];
  const int lane = static_cast<int>(threadIdx.x & 31u), range = w.rec[2];
  const int first = w.index * rg.per, count = min(rg.per, rg.slice_vecs - first);
  if (rg.vec_bytes < 16 || range == kRecordBad || count <= 0) return;
  const int t_lo = range & 0xff, t_hi = range >> 8;
  const auto outside = [&](int id) { return static_cast<unsigned>(id) >= static_cast<unsigned>(p.src_blocks); };
  if constexpr (K == kPlaneToPlane || K == kPlaneToWire || K == kWireToPlane) {
    if (lane != 0 || t_hi - t_lo != p.block_size) return;
    const char* src = rg.src[w.kv];
    if (K == kWireToPlane) {
      const long long before = static_cast<long long>(w.rec[4]) * p.dst_planes + static_cast<long long>(w.plane) * w.rec[5] + w.rec[3];
      const long long image = wire_base(p, w, rg, before, p.block_size);
      if (rg.image_bytes < 16 || image + static_cast<long long>(rg.slice_vecs) * rg.vec_bytes > p.packed_bytes) return;
      src += image;
    } else {
      const int id = w.rec[kRecordHeader + w.plane];
      if (outside(id)) return;
      src += id * rg.block_bytes + rg.slice_at;
    }
    prefetch_l2(src + static_cast<long long>(first) * rg.vec_bytes, count * rg.vec_bytes);
  } else if constexpr (K == kExitToPlane || K == kExitToWire) {
    const int row = first / rg.row_vecs + lane;  // the first 32 rows
    const int begin = max(first, row * rg.row_vecs), end = min(first + count, (row + 1) * rg.row_vecs);
    if (begin >= end) return;
    const int token = p.block_size == 1 ? 0 : row - static_cast<int>(__umulhi(static_cast<unsigned>(row), p.block_magic)) * p.block_size;
    if (token < t_lo || token >= t_hi) return;
    const int e = w.rec[p.exit_at + token];
    if (static_cast<unsigned>(e) >= static_cast<unsigned>(p.src_planes)) return;
    const int id = w.rec[kRecordHeader + e];
    if (outside(id)) return;
    prefetch_l2(rg.src[w.kv] + id * rg.block_bytes + rg.slice_at + static_cast<long long>(begin) * rg.vec_bytes, (end - begin) * rg.vec_bytes);
  }
}

template <typename T, MoveKind K, bool kSplit = false>
__device__ __forceinline__ void move_piece(const MoveParams& p, const MoveRegion& rg, const Piece& w, const PageShared& s, PagePairs& pairs) {
  if constexpr (packs_dedup(K)) {
    pack_pairs<T, kSplit>(p, rg, w, s, pairs);
  } else if constexpr (loops_planes(K)) {
    walk_planes<T, K, kSplit>(p, rg, w, s);
  } else {
    move_rows<T, K, kSplit>(p, rg, w, s);
  }
}

// kAsk: the source is asked for ahead of time.
template <MoveKind K, int kWords, bool kAsk>
__global__ void __launch_bounds__(kThreads, loops_planes(K) ? 3 : 6) move_kernel(const __grid_constant__ MoveArgs<kWords> args) {
  const MoveParams& p = args.p;
  const int* records = kWords > 1 ? args.inline_words : p.records;
  const int* wire = kWords > 1 ? args.inline_words + p.blocks * p.words : p.wire;
  Piece w = piece_at(p, records, blockIdx.x);
  const MoveRegion& rg = p.region[w.g];
  // Records that are parameters may be read before the kernel ahead has ended, and tell where the source is. (Records in device memory would have
  // to be waited for first; asking for pieces further on then costs more than it gives: 29k tokens exit-only 1,758 -> 1,786 us.) Against
  // none: a layer slice of 42 MB 9.1 -> 8.2 us, of 0.2 GB 31.2 -> 29.7; 1,000 tokens exit-only 62.0 -> 60.3 and all planes 234 -> 230.
  if constexpr (kAsk) {
    if (threadIdx.x < 32) prefetch_piece<K>(p, w);
    // (for the rows that exit planes choose, one prefetch each, the pieces ahead are not worth their cost: 60.3 -> 60.5)
    if (!by_token(K) && threadIdx.x / 32 == 1 && gridDim.x - blockIdx.x > kPrefetchAhead)
      prefetch_piece<K>(p, piece_at(p, records, blockIdx.x + kPrefetchAhead));
  }
  follow_stream();
  const int range = w.rec[2];
  if ((packs_dedup(K) || scatters_dedup(K)) && blockIdx.x == 0 && threadIdx.x == 0) {
    p.wire_header[0] = p.wire_tokens;
    p.wire_header[1] = static_cast<long long>(p.blocks) * p.src_planes;
  }
  if (range == kRecordBad) {
    if (threadIdx.x == 0) report(p.status, RLT_STATUS_BAD_RANGE, w.request(), w.rec[3], w.rec[4]);
    return;
  }
  w.t_lo = range & 0xff;
  w.t_hi = range >> 8;
  __shared__ PageShared shared;  // not allocated where nothing touches it
  __shared__ PagePairs pairs;
  if constexpr (loops_planes(K) || K == kExitToPlane || K == kExitToWire || packs_dedup(K))
    fetch_page<K>(p, rg, w, wire + (w.rec - records) / p.words * p.src_planes, shared);
  if (rg.vec_bytes == 32) {
    move_piece<Vec32, K>(p, rg, w, shared, pairs);
  } else if (rg.vec_bytes == 16) {
    if constexpr (K == kPlaneToWire || K == kExitToWire || K == kWireToPlane || K == kDedupToOddWire || K == kDedupFromOddWire) {
      if (rg.image_bytes < 16) return move_piece<uint4, K, true>(p, rg, w, shared, pairs);
    }
    move_piece<uint4, K>(p, rg, w, shared, pairs);
  } else if (rg.vec_bytes == 4) {
    move_piece<uint32_t, K>(p, rg, w, shared, pairs);
  } else {
    move_piece<uint8_t, K>(p, rg, w, shared, pairs);
  }
}

template <MoveKind K, int kWords>
cudaError_t launch_move(const MoveParams& p, const RltBlockMoves& m, unsigned grid, bool ask, cudaStream_t stream) {
  MoveArgs<kWords> args;
  args.p = p;
  if (kWords > 1) {
    const size_t n = static_cast<size_t>(m.blocks) * m.words;
    std::memcpy(args.inline_words, m.host_records, n * sizeof(int));
    if (m.host_wire != nullptr)
      std::memcpy(args.inline_words + n, m.host_wire, static_cast<size_t>(m.blocks) * p.src_planes * sizeof(int));
  }
  if constexpr (kWords > 1 && asks_ahead(K)) {
    if (asking(ask)) return launch_following(move_kernel<K, kWords, true>, grid, kThreads, stream, args);
  }
  return launch_following(move_kernel<K, kWords, false>, grid, kThreads, stream, args);
}

// int32 that the launch's parameters would have to hold.
long long parameter_words(const MoveParams& p, const RltBlockMoves& m) {
  return static_cast<long long>(m.blocks) * m.words + (m.host_wire ? static_cast<long long>(m.blocks) * p.src_planes : 0);
}

template <MoveKind K>
int launch_kind(const MoveParams& p, const RltBlockMoves& m, unsigned grid, bool ask, cudaStream_t stream) {
  const long long n = parameter_words(p, m);
  // A parameter block is copied into the launch whole (a launch takes the host 1.85 us with 0.1 - 7 KiB, 2.2 with 16 and 3.1 with 31; a
  // copy of the records, the launch and an event 4.5, and the GPU 9 - 16 us more), so three sizes of it: the small one covers a few
  // hundred tokens, the medium one a thousand.
  cudaError_t launched;
  if (n <= kInlineSmallWords) {
    launched = launch_move<K, kInlineSmallWords>(p, m, grid, ask, stream);
  } else if (n <= kInlineMediumWords) {
    launched = launch_move<K, kInlineMediumWords>(p, m, grid, ask, stream);
  } else if (n <= kInlineWords) {
    launched = launch_move<K, kInlineWords>(p, m, grid, ask, stream);
  } else if (p.records != nullptr && (m.host_wire == nullptr || p.wire != nullptr)) {
    launched = launch_move<K, 1>(p, m, grid, ask, stream);
  } else {
    return RLT_E_INVALID;
  }
  RLT_CUDA_TRY(launched);
  return RLT_OK;
}

int vectors_per_round(int vec_bytes, bool planes) {
  return kThreads * (vec_bytes == 32 ? unroll_of<Vec32>(planes) : vec_bytes == 16 ? unroll_of<uint4>(planes)
                     : vec_bytes == 4 ? unroll_of<uint32_t>(planes) : unroll_of<uint8_t>(planes));
}

// How the pairs of a page are dealt to CTAs in a dedup pack. What the pages contribute is known, and the average is cut: a layer's pairs into a power
// of two of shares, or whole layers put together, so that shares of an average page end where layers do. The first of these cuts that gives the GPU
// enough CTAs is taken: the most that a share holds, in eighths of a round of 16 KiB, and the waves of six CTAs per SM that are enough.
//
// Every CTA first lists its page's pairs, so shares below 64 KiB lose more than a fuller GPU gains: 5 prompts on four planes, shares of 160 / 80 / 53 / 40 /
// 32 KiB, 850 / 843 / 911 / 922 / 1,011 us. Three and seven shares a layer are worse than two and four: all tokens of 6 prompts on four planes, 2 / 3 / 4
// shares 984 / 1,010 / 1,011; 16 planes, 4 / 7 / 8 shares 661 / 674 / 663. A launch of few waves is better with smaller ones: 700 tokens on four planes
// (4.8 waves of 80 KiB) 115 -> 111 with 40 KiB; 2,500 on one plane (8.5 of 64) 153 -> 148 with 32, but 5,000 (17 of 64) stay; 300 on six planes (4.1 of 56)
// 73 with 28 KiB, 71 when they stay; 100 on four (1.5 of 36) 24 with 18 KiB, 19.5 when they stay. Rows below 1 KiB take a CTA longer than larger ones do: 352 pages of
// 384-byte rows on seven planes (4.8 waves of 120 KiB) 185 with shares of 48 KiB, 178 when they stay.
//
// Pages that contribute much more than the average get longer shares. More shares for every page, until the deepest one's are short, is
// far worse (16 planes, 450 pages on one plane and 20 on all: 733 us so, 1,247 with at most twice the average's share, 1,924 with
// at most its own; 1,330 where every page had the shares of a full one).
struct PackCut {
  int eighths, waves, waves_of_short_rows;
};
constexpr PackCut kPackCuts[] = {{70, 8, 4}, {35, 12, 12}, {30, 1, 1}, {15, 0, 0}};
constexpr int kShortRow = 1024;

int pack_shares(const MoveRegion& rg, const MoveParams& p, const RltBlockMoves& m, const PackCut& cut) {
  const long long layer = std::max<long long>(1, rg.row_vecs * ((m.wire_tokens + m.blocks - 1) / m.blocks));
  const long long most = vectors_per_round(rg.vec_bytes, false) * cut.eighths / 8;
  long long count = p.slice_layers;
  if (layer > most) {
    for (long long share = layer; share > most; share = (share + 1) / 2) count *= 2;
  } else {
    const long long layers = most / layer;
    count = (count + layers - 1) / layers;
  }
  // no share of a full page may have more vectors than the multiplier split of pack_pairs allows
  return static_cast<int>(std::max(count, (static_cast<long long>(rg.slice_vecs) * p.src_planes + 65535) / 65536));
}

// Whether a launch of a kind that can ask for its source does.
bool asks(const MoveParams& p, const RltBlockMoves& m, MoveKind kind, int regions) {
  if (parameter_words(p, m) > kInlineWords) return false;  // records in device memory would have to be waited for (move_kernel)
  long long bytes = 0;
  for (int g = 0; g < regions; ++g) bytes += 4ll * m.blocks * p.grid_planes * p.region[g].slice_vecs * p.region[g].vec_bytes;
  if (bytes < kPrefetchBytes) return false;
  if (by_token(kind)) {
    // A prefetch per row costs a long launch more than the start of it gains. Exit-only handoffs one behind another, us without / with it: 39 MB
    // 6.7 / 6.6, 79 MB 11.9 / 11.0, 0.20 GB 30.8 / 29.2, 0.39 GB 60.8 / 59.1, 0.47 GB 73.4 / 73.7, 0.59 GB 90.6 / 90.7, 1.2 GB 178.7 / 180.1.
    if (bytes > (448ll << 20)) return false;
  } else {
    // Where all rows of a page come from one place, only pages that are wholly in range are asked for, and the blocks of the others partly idle.
    // Much of that and asking costs more than it gives. Prompts of two pages of 4 KiB rows, us without / with it, by the share of the pages' tokens that
    // is in range: handoffs, 32-token pages, 0.55 983 / 1,021, 0.65 930 / 946, 0.75 921 / 911, 0.85 923 / 912; 64-token pages, 0.51 708 / 727, 0.72 799 / 801,
    // 0.75 901 / 889; 16-token pages, 0.53 120.1 / 121.6, 0.75 558 / 552. Packs 0.55 1,003 / 1,053, 0.65 927 / 950, 0.75 912 / 906, but in 64-token pages
    // 0.75 894 / 905 and 0.85 912 / 904; scatters like packs. FP8 in 16-token pages, 0.56 433 / 441, 0.75 578 / 569.
    long long used = 0;
    for (int b = 0; b < m.blocks; ++b) {
      const int range = m.host_records[static_cast<size_t>(b) * m.words + 2];
      if (range != kRecordBad) used += (range >> 8) - (range & 0xff);
    }
    if (4 * used < 3ll * m.blocks * p.block_size) return false;
  }
  // every tensor that is asked for (an image: once)
  for (int g = 0; g < regions; ++g) {
    const MoveRegion& rg = p.region[g];
    if (rg.vec_bytes < 16) continue;
    if (!prefetches(rg.src[0], bytes)) return false;
    if (kind == kWireToPlane) break;
    if (!prefetches(rg.src[1], bytes)) return false;
  }
  return true;
}

}  // namespace
}  // namespace rlt

extern "C" int rlt_move_blocks(int direction, const RltPool* src, const RltPool* dst, const RltBlockMoves* m,
                               const RltOptions* opt, void* packed, int64_t packed_bytes, rlt_stream_t stream) {
  using namespace rlt;
  const Direction dir = static_cast<Direction>(direction);
  const NvtxRange range(dir == kDirect ? "rlt.kv_handoff" : dir == kPack ? "rlt.kv_pack" : "rlt.kv_scatter");
  if (m == nullptr || opt == nullptr) return RLT_E_INVALID;
  // The checks of the table-driven entry points, on a batch of the same shape (its arrays are never touched).
  static const int32_t present = 0;
  static const int64_t present64 = 0;
  RltBatch shape = {};
  shape.num_requests = m->num_requests;
  shape.table_width = m->table_width;
  shape.src_tables = m->src_planes ? &present : nullptr;
  shape.dst_tables = m->dst_planes ? &present : nullptr;
  shape.tok_begin = shape.tok_end = &present;
  if (m->has_exit) {
    shape.exit_planes = &present;
    shape.exit_offsets = &present64;
    shape.exit_count = 1;
  }
  TableCopyParams t;
  const int checked = table_params(dir, src, dst, &shape, opt, packed, packed_bytes, t);
  if (checked != RLT_OK) return checked;
  const bool dedup = opt->mode == RLT_MODE_DEDUP;
  if (t.dedup_wire) {
    if (opt->workspace == nullptr) return RLT_E_INVALID;
    if (reinterpret_cast<uintptr_t>(opt->workspace) & 15u) return RLT_E_ALIGN;
    if (opt->workspace_bytes < dedup_workspace_bytes(m->num_requests, m->table_width, t.src_planes)) return RLT_E_LIMIT;
  }
  if (opt->variant != 0 || opt->grid_limit != 0 || t.src_planes > kMaxPlanes || t.dst_planes > kMaxPlanes) return RLT_MOVE_UNSUITED;
  if (dir != kDirect && (t.plane_begin != 0 || t.plane_count != t.dst_planes)) return RLT_MOVE_UNSUITED;
  if (t.block_size != m->block_size || (dir != kScatter && m->src_planes != t.src_planes) ||
      (dir != kPack && m->dst_planes != t.dst_planes))
    return RLT_MOVE_UNSUITED;
  // a CTA lists a page's blocks on both sides, also on the one that this direction does not touch
  if (m->src_planes > kMaxPlanes || m->dst_planes > kMaxPlanes) return RLT_MOVE_UNSUITED;
  if (t.dedup_wire && m->host_wire == nullptr) return RLT_MOVE_UNSUITED;
  if (m->blocks == 0) return RLT_OK;

  MoveKind kind = dir == kDirect ? (dedup ? kFanOut : opt->mode == RLT_MODE_EXIT_ONLY ? kExitToPlane : kPlaneToPlane)
                        : dir == kPack ? (dedup ? kDedupToWire : opt->mode == RLT_MODE_EXIT_ONLY ? kExitToWire : kPlaneToWire)
                                       : (dedup ? kDedupFromWire : kWireToPlane);
  const bool planes = loops_planes(kind), pairs = packs_dedup(kind);
  MoveParams p = {};
  p.slice_layers = t.layer_end - t.layer_begin;
  for (int g = 0; g < t.num_regions; ++g) {
    const RegionParams& s = t.region[g];
    MoveRegion& rg = p.region[g];
    rg.src[0] = s.src_key;
    rg.src[1] = s.src_value;
    rg.dst[0] = s.dst_key;
    rg.dst[1] = s.dst_value;
    rg.block_bytes = s.block_bytes;
    rg.slice_at = s.layer_bytes * t.layer_begin;
    rg.token_bytes = static_cast<int>(s.token_bytes);
    // of the pool's side; the image's rows lie on multiples of the largest power of two that divides all sizes in it
    const uintptr_t rows_at = static_cast<uintptr_t>(s.token_bytes) | (dir == kScatter ? 0 : reinterpret_cast<uintptr_t>(s.src_key) | reinterpret_cast<uintptr_t>(s.src_value)) |
                              (dir == kPack ? 0 : reinterpret_cast<uintptr_t>(s.dst_key) | reinterpret_cast<uintptr_t>(s.dst_value));
    uintptr_t image_at = dir == kDirect ? 0 : reinterpret_cast<uintptr_t>(packed);
    for (int h = 0; dir != kDirect && h < t.num_regions; ++h) image_at |= static_cast<uintptr_t>(t.region[h].token_bytes);
    rg.image_bytes = image_at & 4u ? 4 : image_at & 8u ? 8 : 16;
    rg.vec_bytes = (rows_at | image_at) & 3u ? 1 : ((rows_at | image_at) & 31u) == 0 ? 32 : (rows_at & 15u) == 0 ? 16 : 4;
    if (rg.vec_bytes == 16 && rg.image_bytes < 16 && t.dedup_wire) kind = dir == kPack ? kDedupToOddWire : kDedupFromOddWire;
    const long long row_vecs = s.token_bytes / rg.vec_bytes;
    const long long slice_vecs = row_vecs * t.block_size * p.slice_layers;
    // the multiplier splits of row_at: (row_vecs + piece) * row_vecs and rows * block_size below 2^32
    if ((row_vecs + 65536) * row_vecs >= (1ll << 32) || slice_vecs * t.src_planes >= (1ll << 30) ||
        static_cast<long long>(t.block_size) * t.block_size * p.slice_layers >= (1ll << 32))
      return RLT_MOVE_UNSUITED;
    // the one of pack_pairs: (layers x pairs of a page) * pairs
    const long long most_pairs = static_cast<long long>(t.block_size) * t.src_planes;
    if (pairs && most_pairs * most_pairs * p.slice_layers >= (1ll << 32)) return RLT_MOVE_UNSUITED;
    rg.row_vecs = static_cast<int>(row_vecs);
    rg.row_magic = row_vecs == 1 ? 0u : div_magic(static_cast<uint32_t>(row_vecs));
    rg.slice_vecs = static_cast<int>(slice_vecs);
  }
  p.plane_begin = t.plane_begin;
  p.plane_end = t.plane_begin + t.plane_count;
  p.grid_planes = planes || pairs ? 1 : t.plane_count;
  p.src_planes = t.src_planes;
  p.dst_planes = t.dst_planes;
  p.src_blocks = t.src_blocks;
  p.dst_blocks = t.dst_blocks;
  p.block_size = t.block_size;
  p.block_magic = t.block_size == 1 ? 0u : div_magic(static_cast<uint32_t>(t.block_size));
  p.layer_begin = t.layer_begin;
  p.deep_layer_mask = t.deep_layer_mask;
  p.packed_bytes = t.packed_bytes;
  p.packed_token_bytes = t.packed_token_bytes;
  p.words = m->words;
  p.blocks = m->blocks;
  p.dst_at = kRecordHeader + m->src_planes;
  p.exit_at = kRecordHeader + m->src_planes + m->dst_planes;
  p.records = m->device_records;
  p.wire = m->device_wire;
  p.wire_header = static_cast<long long*>(opt->workspace);
  p.wire_tokens = m->wire_tokens;
  p.status = opt->status;
  // Rounds of a piece. Where a plane's block is all a CTA looks up, one: the smaller the piece the closer the SMs stay
  // together. Kinds that fetch the page's record and work out exit planes first need more payload behind that: measured
  // best at 2 for exit-only (29k tokens: 1.84 -> 1.75 ms); a dedup pack has a rule of its own (pack_shares). Where planes are walked, the
  // more planes a round stores to the fewer rounds are needed, 12 / planes and at most 4. Dedup handoffs of 6 - 8.6 GB, us at
  // 1 / 2 / 3 / 4 / 8 rounds: two planes 1,267 / 1,105 / 1,054 / 1,026 / 991 (so 8 would be 4 % faster there), three 1,199 /
  // 1,093 / 1,053 / 1,036 / 1,039, four 1,295 / 1,234 / 1,226 / 1,227 / 1,240, six 1,289 / 1,270 / 1,267 / 1,270 / 1,281, eight
  // 1,185 / 1,190 / 1,191 / 1,196 / 1,205, sixteen 1,282 / 1,295 / 1,298 / 1,307 / 1,321, 32 1,086 / 1,098 / 1,105 / 1,114 /
  // 1,114; scatters of dedup images within 1 % of the same. A launch of fewer than eight waves takes the smallest piece that a
  // larger one would split into: it is short of CTAs, not of payload per CTA.
  int sms = 0;
  const int found = sm_count(&sms);
  if (found != RLT_OK) return found;
  int rounds = planes ? std::max(1, std::min(4, 12 / p.dst_planes)) : by_token(kind) ? 2 : 1;
  const PackCut* cut = kPackCuts;  // the last of them ends the search
  long long grid = 0;
  for (;;) {
    p.pieces = 0;
    for (int g = 0; g < t.num_regions; ++g) {
      MoveRegion& rg = p.region[g];
      rg.per = vectors_per_round(rg.vec_bytes, planes) * rounds;
      rg.pieces = pairs ? pack_shares(rg, p, *m, *cut) : (rg.slice_vecs + rg.per - 1) / rg.per;
      p.pieces += 2 * rg.pieces;
    }
    grid = static_cast<long long>(m->blocks) * p.grid_planes * p.pieces;
    const long long wave = static_cast<long long>(sms) * (planes ? 3 : 6);
    if (pairs) {
      if (grid >= wave * (p.region[0].token_bytes < kShortRow ? cut->waves_of_short_rows : cut->waves)) break;
      ++cut;
    } else {
      if (rounds == 1 || grid >= 8 * wave) break;
      rounds /= 2;
    }
  }
  if (grid > 0x7fffffffll) return RLT_MOVE_UNSUITED;
  const bool ask = asks_ahead(kind) && asks(p, *m, kind, t.num_regions);

  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const unsigned ctas = static_cast<unsigned>(grid);
  int rc = RLT_E_INVALID;
  switch (kind) {
    case kPlaneToPlane: rc = launch_kind<kPlaneToPlane>(p, *m, ctas, ask, s); break;
    case kExitToPlane: rc = launch_kind<kExitToPlane>(p, *m, ctas, ask, s); break;
    case kFanOut: rc = launch_kind<kFanOut>(p, *m, ctas, ask, s); break;
    case kPlaneToWire: rc = launch_kind<kPlaneToWire>(p, *m, ctas, ask, s); break;
    case kExitToWire: rc = launch_kind<kExitToWire>(p, *m, ctas, ask, s); break;
    case kDedupToWire: rc = launch_kind<kDedupToWire>(p, *m, ctas, ask, s); break;
    case kWireToPlane: rc = launch_kind<kWireToPlane>(p, *m, ctas, ask, s); break;
    case kDedupFromWire: rc = launch_kind<kDedupFromWire>(p, *m, ctas, ask, s); break;
    case kDedupToOddWire: rc = launch_kind<kDedupToOddWire>(p, *m, ctas, ask, s); break;
    case kDedupFromOddWire: rc = launch_kind<kDedupFromOddWire>(p, *m, ctas, ask, s); break;
  }
  if (rc != RLT_OK) return rc;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

extern "C" int rlt_load_moves(void) {
  using namespace rlt;
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, kInlineSmallWords, true>));
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, kInlineSmallWords, false>));
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, kInlineMediumWords, true>));
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, kInlineMediumWords, false>));
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, kInlineWords, true>));
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, kInlineWords, false>));
  RLT_CUDA_TRY(load_kernel(move_kernel<kPlaneToPlane, 1, false>));
  return RLT_OK;
}
