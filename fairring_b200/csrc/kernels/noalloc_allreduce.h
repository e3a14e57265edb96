// An entry point for callers that are not allowed to allocate.
//
// This function has no counterpart in the reference.  It exists for hosts of
// this library that must not call cudaMalloc (or anything that does) at the
// moment they need a reduction: code running while a CUDA graph is being
// captured elsewhere in the process, plugins living inside another runtime's
// memory budget, real-time loops where an allocation may stall behind the
// driver's lock.  Everything else in this library gets its staging memory from
// the engine at start-up; this needs no staging at all.
#pragma once

#ifdef __cplusplus
extern "C" {
#endif

// Sums `world` fp32 buffers of `numel` elements element-wise, in the order of
// `bufs`, and leaves the sum in every one of them (an all-reduce whose ranks
// are buffers on the current device).
//
//   bufs    host array of `world` device pointers (fp32, `numel` elements each,
//           on the current device -- checked; the buffers must not overlap).
//           16-byte aligned buffers are read four elements at a time.
//   world   2..8
//   numel   1..4096
//   stream  a cudaStream_t of the current device (0 for the default stream)
//   check   non-zero: wait for the stream and report its errors
//   err     optional buffer that receives a message when the call fails
//
// Returns 0 on success, 1 for a bad argument (too many buffers, too many
// elements, null pointer: nothing has been launched), 2 for a CUDA error.
//
// Calls no cudaMalloc/cudaFree and no allocating library routine; one kernel
// launch, nothing else on the stream.  Nothing is kept between calls: calls on
// different streams and from different threads do not disturb each other.
int fairring_allreduce_f32_noalloc(float* const* bufs, int world, long long numel, void* stream,
                                   int check, char* err, unsigned long err_len);

#ifdef __cplusplus
}
#endif
