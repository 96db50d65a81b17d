// Entry points between the library and its own Python module: not part of the C ABI.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include "rlt_kv_handoff.h"

#ifdef __cplusplus
extern "C" {
#endif

// Copies `bytes` bytes of ordinary host memory to the current device through a pinned buffer of the library, on `stream`;
// the host memory is free again on return. On a stream that is capturing a graph the buffer belongs to that graph for as long as it
// lives: every replay copies it again.
RLT_API int rlt_stage_upload(const void* host, size_t bytes, void* device, rlt_stream_t stream);
RLT_API int rlt_capture_id(rlt_stream_t stream, uint64_t* id);  // of the capture that `stream` takes part in; 0: none

// rlt_tensor_transfer between tensors of one type, with the descriptor table in HOST memory: it travels as kernel
// parameters, so nothing has to be kept for the launch. At most RLT_INLINE_TRANSFERS descriptors.
#define RLT_INLINE_TRANSFERS 448
RLT_API int rlt_tensor_transfer_inline(const int64_t* descriptors, int32_t count, int32_t max_rows, int32_t max_cols,
                                       int32_t dtype, rlt_stream_t stream);

// How many launches of this process have asked L2 for their source ahead of time, and how many addresses were looked up for that.
RLT_API void rlt_prefetch_counts(int64_t counts[2]);

// rlt_kv_post behind copies of a few small byte ranges, (source, destination, bytes) in HOST memory, in one launch.
#define RLT_POST_RANGES 4
#define RLT_POST_RANGE_BYTES 32768  // of all of them
RLT_API int rlt_post_behind(const int64_t* ranges, int32_t count, void* slot, const uint8_t body[56], uint64_t stamp, rlt_stream_t stream);

// Loads what a transfer worker launches, on the current device, for pools of so many planes. The kernels of a source file are otherwise loaded by the
// first launch of any of them, and that waits for what runs on the device by then: a message that should be queued behind a prefill would
// hold the host until the prefill has ended. (The other kernels of a file do not wait once one of them has been loaded.)
RLT_API int rlt_load_transport(int32_t planes);
int rlt_load_tables(void);
int rlt_load_moves(void);
int rlt_load_segments(void);

// rlt_kv_copy_segments with the (source, destination, bytes) triples in HOST memory: they travel as kernel parameters.
#define RLT_INLINE_SEGMENTS 1024
RLT_API int rlt_copy_segments_inline(const int64_t* triples, int32_t count, rlt_stream_t stream);

// Events of the current device that outlive the objects using them: taken from a pool, recorded on `stream`, given back. An
// event that is given back before it has fired may be recorded again at once: nobody looks at it any more.
typedef struct RltEvent RltEvent;
RLT_API int rlt_event_record(int timed, rlt_stream_t stream, RltEvent** out);
RLT_API int rlt_event_query(RltEvent* event);  // 1: fired, 0: not yet, negative: RLT_E_*
RLT_API int rlt_event_wait(RltEvent* event);   // on the host
RLT_API int rlt_event_order(RltEvent* event, rlt_stream_t stream);  // what is queued on `stream` from now on comes after it
RLT_API int rlt_event_elapsed(RltEvent* from, RltEvent* to, float* milliseconds);
RLT_API void rlt_event_release(RltEvent* event);

#ifdef __cplusplus
}
#endif
