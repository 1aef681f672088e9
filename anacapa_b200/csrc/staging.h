// Copies between host memory and the device, of pageable memory through pinned
// chunks.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace ana {

// Large copies of pageable memory run on a few threads, each with its own stream
// and two pinned chunks: one chunk crosses the bus while the other is copied from
// or to the caller's memory, whose pages are often touched there for the first
// time. The driver's own path for pageable memory does both in turn on one
// thread. Memory that it moves directly (page-locked, managed) and short copies
// are left to it.
//
// Sets of chunks (1 MiB pinned, 8 MiB more once a set has copied 128 MiB),
// streams and events are shared by the contexts of a process: a copy takes an
// idle set of its device, or makes one (1-3 milliseconds), and gives it back. Two idle sets at most are kept per device,
// and none once the device's last context is gone.

// Every context holds one reference (stage_retain at its creation).
void stage_retain(int device);
void stage_release(int device);

// dst (host) <- src (device), after the work queued on st. Complete on return.
cudaError_t stage_read(void* dst, const void* src, size_t bytes, cudaStream_t st, int device);
// dst (device) <- src (host), after the work queued on st and before what is
// queued on it later. Pageable src may be reused on return, page-locked src once
// st has passed the copy.
cudaError_t stage_write(void* dst, const void* src, size_t bytes, cudaStream_t st, int device);

}  // namespace ana
