// Allocation-free AllReduce over buffers that live on ONE GPU.
//
// This entry point has no counterpart in the reference library.
//
// Who it is for: callers that hold several same-sized buffers on one device
// (per-micro-batch gradient replicas, per-expert partial results, the virtual
// ranks of a single-process test) and must combine them from a place where
// device memory cannot be allocated or freed: inside a region where the
// framework's allocator is locked or its pool is exhausted on purpose, in a
// library that promised its host application a fixed memory footprint, or in
// code that runs while the driver refuses allocation calls (for instance while
// another thread captures a stream in global capture mode).  Those callers
// cannot use mncclEmuCreate / mncclEmuCollective, which cudaMalloc the control
// segments, inboxes and the parameter table.
//
// What it does: one kernel that reads every buffer, reduces in buffer order (fp32 accumulation for the
// floating types, the bits of the one-shot collective kernel) and writes every result.  Pointers travel by
// value; no cudaMalloc, cudaFree or allocating library routine is called, in set-up or later, and no
// state is kept between calls except the two words of the outcome record, a `static __device__` array.
//
// Limits (requests beyond them are rejected with ncclInvalidArgument and a
// message): 2..kNoAllocMaxRanks buffers, at most kNoAllocMaxBytes bytes each;
// types fp32, fp16, bf16, int32; operators sum, prod, max, min, avg.
//
// send[r] may equal recv[r'] for any r, r'; buffers that overlap otherwise race.  Calls on different
// streams do not disturb one another.
#pragma once
#include <stddef.h>

#include "mini_nccl_api.h"

#ifdef __cplusplus
extern "C" {
#endif

enum { kNoAllocMaxRanks = 4 };
enum { kNoAllocMaxBytes = 64 * 1024 };

/* recv[r][i] = scale-free reduction over r' of send[r'][i], for every r.
 * send / recv: `nbuffers` device pointers each (host arrays of pointers); send[r] may equal recv[r]. */
ncclResult_t mncclLocalAllReduceNoAlloc(const void* const* send, void* const* recv, int nbuffers, size_t count,
                                        ncclDataType_t datatype, ncclRedOp_t op, cudaStream_t stream);

/* Size in bytes of the static device memory (per GPU): the outcome record. */
size_t mncclNoAllocScratchBytes(void);

/* Outcome of the last call on the current device: *status 0 (and *detail 0, may be NULL) when its kernel
 * completed.  The kernel waits for nothing, so a call that was launched has no other outcome; the entry point
 * stays for callers of earlier versions.  Synchronises `stream`, reads eight bytes, allocates nothing. */
ncclResult_t mncclNoAllocLastStatus(cudaStream_t stream, unsigned* status, unsigned* detail);

#ifdef __cplusplus
}
#endif
