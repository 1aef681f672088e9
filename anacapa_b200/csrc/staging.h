// Copies between pageable host memory and the device through pinned chunks.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace ana {

// One per context (one caller at a time, like the context). Large copies run on
// a few threads, each with its own stream and two pinned chunks: one chunk
// crosses the bus while the other is copied from or to the caller's memory,
// whose pages are often touched there for the first time. The driver's own
// path for pageable memory does both in turn on one thread. Chunks, streams and
// events (8 MiB pinned) are made at the first large copy and kept until
// release().
class HostStage {
public:
    ~HostStage() { release(); }
    void release();
    // dst (host) <- src (device), after the work queued on st. Complete on return.
    cudaError_t read(void* dst, const void* src, size_t bytes, cudaStream_t st, int device) {
        return copy(dst, src, bytes, st, device, true);
    }
    // dst (device) <- src (host), after the work queued on st and before what
    // is queued on it later. src may be reused on return.
    cudaError_t write(void* dst, const void* src, size_t bytes, cudaStream_t st, int device) {
        return copy(dst, src, bytes, st, device, false);
    }

private:
    static constexpr int kThreads = 4;
    static constexpr size_t kChunk = size_t(1) << 20;
    cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t st, int device, bool out);
    bool ensure();
    cudaError_t run(int t, int threads, unsigned char* dst, const unsigned char* src, size_t bytes, int device, bool out);
    unsigned char* pinned_ = nullptr;
    cudaStream_t stream_[kThreads] = {};
    cudaEvent_t done_[kThreads][2] = {};
    cudaEvent_t begin_ = nullptr;
    bool failed_ = false;
};

}  // namespace ana
