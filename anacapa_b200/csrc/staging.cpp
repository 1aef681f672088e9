#include "staging.h"

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>

namespace ana {

namespace {

class HostStage {
public:
    explicit HostStage(int device) : device_(device) {}
    ~HostStage();
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;
    int device() const { return device_; }
    bool make();  // on the current device; false: no pinned memory to be had
    cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t st, bool out);

private:
    static constexpr int kThreads = 4;
    // Page-locking a set is part of the first large copy of a program's only
    // context: 8 MiB takes 4-10 ms, 1 MiB 1-2.6. Copies through 128 KiB chunks
    // (1 MiB a set) are slower: a 1920x1080 film into used pages takes 3.06 ms,
    // through 1 MiB chunks 1.6, through the driver's own path 2.35; 960x540 0.87,
    // 0.45, 0.60; 2^20 rays and hits 4.9, 2.4, 4.6. That is 8 MiB's cost for
    // every 128-256 MiB copied, so a set that has copied kGrowAfter takes the
    // larger chunks: no program pays much more than twice the better choice.
    static constexpr size_t kSmallChunk = size_t(1) << 17, kLargeChunk = size_t(1) << 20;
    static constexpr size_t kGrowAfter = size_t(128) << 20;
    void grow();
    cudaError_t run(int t, int threads, unsigned char* dst, const unsigned char* src, size_t bytes, bool out);
    int device_;
    unsigned char* pinned_ = nullptr;  // the chunks in use
    unsigned char* small_ = nullptr;   // the first ones: freeing them may wait for the device
    unsigned char* large_ = nullptr;
    size_t chunk_ = kSmallChunk, copied_ = 0;
    cudaStream_t stream_[kThreads] = {};
    cudaEvent_t done_[kThreads][2] = {};
    cudaEvent_t begin_ = nullptr;
};

// Copies below this take the driver's path: the threads cost more than they
// save (0.1-0.2 ms for starting and joining them).
constexpr size_t kStageMin = size_t(1) << 20;

HostStage::~HostStage() {
    for (int t = 0; t < kThreads; ++t) {
        if (stream_[t]) cudaStreamDestroy(stream_[t]);
        for (cudaEvent_t e : done_[t])
            if (e) cudaEventDestroy(e);
    }
    if (begin_) cudaEventDestroy(begin_);
    if (small_) cudaFreeHost(small_);
    if (large_) cudaFreeHost(large_);
}

bool HostStage::make() {
    void* p = nullptr;
    bool ok = cudaHostAlloc(&p, kThreads * 2 * kSmallChunk, cudaHostAllocPortable) == cudaSuccess;
    if (ok) pinned_ = small_ = static_cast<unsigned char*>(p);
    ok = ok && cudaEventCreateWithFlags(&begin_, cudaEventDisableTiming) == cudaSuccess;
    for (int t = 0; ok && t < kThreads; ++t) {
        ok = cudaStreamCreateWithFlags(&stream_[t], cudaStreamNonBlocking) == cudaSuccess;
        for (cudaEvent_t& e : done_[t]) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) cudaGetLastError();
    return ok;
}

// Without memory for it, asked again after as much has been copied.
void HostStage::grow() {
    copied_ = 0;
    void* p = nullptr;
    if (cudaHostAlloc(&p, kThreads * 2 * kLargeChunk, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    pinned_ = large_ = static_cast<unsigned char*>(p);
    chunk_ = kLargeChunk;
}

// Thread t's chunks t, t + threads, ...
cudaError_t HostStage::run(int t, int threads, unsigned char* dst, const unsigned char* src, size_t bytes, bool out) {
    cudaError_t e = cudaSetDevice(device_);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream_[t], begin_, 0);
    const size_t chunks = (bytes + chunk_ - 1) / chunk_, step = size_t(threads);
    unsigned char* slot[2] = {pinned_ + size_t(2 * t) * chunk_, pinned_ + size_t(2 * t + 1) * chunk_};
    auto size_of = [&](size_t k) { return std::min(chunk_, bytes - k * chunk_); };
    auto fetch = [&](size_t k, int s) {
        cudaError_t r = cudaMemcpyAsync(slot[s], src + k * chunk_, size_of(k), cudaMemcpyDeviceToHost, stream_[t]);
        return r == cudaSuccess ? cudaEventRecord(done_[t][s], stream_[t]) : r;
    };
    int s = 0;
    if (out) {
        if (e == cudaSuccess && size_t(t) < chunks) e = fetch(size_t(t), 0);
        for (size_t k = size_t(t); e == cudaSuccess && k < chunks; k += step, s ^= 1) {
            if (k + step < chunks) e = fetch(k + step, s ^ 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(done_[t][s]);
            if (e == cudaSuccess) std::memcpy(dst + k * chunk_, slot[s], size_of(k));
        }
    } else {
        for (size_t k = size_t(t), i = 0; e == cudaSuccess && k < chunks; k += step, ++i, s ^= 1) {
            if (i >= 2) e = cudaEventSynchronize(done_[t][s]);  // the slot's last copy has left it
            if (e != cudaSuccess) break;
            std::memcpy(slot[s], src + k * chunk_, size_of(k));
            e = cudaMemcpyAsync(dst + k * chunk_, slot[s], size_of(k), cudaMemcpyHostToDevice, stream_[t]);
            if (e == cudaSuccess) e = cudaEventRecord(done_[t][s], stream_[t]);
        }
    }
    const cudaError_t f = cudaStreamSynchronize(stream_[t]);  // the slots are free for the next copy
    return e == cudaSuccess ? f : e;
}

// Into fresh pages the driver's own path takes 8.9 ms for a 1920x1080 film (41 MB)
// and 9.7 for 2^20 rays and hits (32 MB each) with their traversal; small chunks
// 4.0 and 5.9, large ones 2.7-3.4 and 3.8-4.2.
cudaError_t HostStage::copy(void* dst, const void* src, size_t bytes, cudaStream_t st, bool out) {
    if (!large_ && copied_ >= kGrowAfter) grow();
    copied_ += bytes;
    cudaError_t e = cudaEventRecord(begin_, st);
    if (e != cudaSuccess) return e;
    const unsigned cores = std::thread::hardware_concurrency();
    const int threads = int(std::min<size_t>({size_t(kThreads), std::max<size_t>(1, cores / 2), (bytes + chunk_ - 1) / chunk_}));
    cudaError_t result[kThreads] = {};
    auto work = [&](int t) {
        result[t] = run(t, threads, static_cast<unsigned char*>(dst), static_cast<const unsigned char*>(src), bytes, out);
    };
    std::thread pool[kThreads];
    int started = 1;
    try {
        for (; started < threads; ++started) pool[started] = std::thread(work, started);
    } catch (...) {  // no thread or no memory for one to be had: this one does their part
    }
    work(0);
    for (int t = started; t < threads; ++t) work(t);
    for (int t = 1; t < started; ++t) pool[t].join();
    for (int t = 0; t < threads; ++t)
        if (result[t] != cudaSuccess) e = result[t];
    return e;
}

// The sets not in use, by device: a copy of another device's context finds its
// own idle. Never destroyed itself (at the process's end the driver may be gone
// before it), and nothing in it allocates.
constexpr int kDevices = 64;  // sets of higher ordinals are made for each copy
constexpr int kIdle = 2;
struct Pool {
    std::mutex mu;
    struct {
        int contexts = 0;
        std::unique_ptr<HostStage> idle[kIdle];
    } dev[kDevices];
};
Pool& pool() {
    alignas(Pool) static unsigned char mem[sizeof(Pool)];
    static Pool* p = new (mem) Pool;
    return *p;
}

std::unique_ptr<HostStage> take(int device) {
    if (device < kDevices) {
        std::lock_guard<std::mutex> lk(pool().mu);
        for (std::unique_ptr<HostStage>& s : pool().dev[device].idle)
            if (s) return std::move(s);
    }
    std::unique_ptr<HostStage> s(new (std::nothrow) HostStage(device));
    if (s && !s->make()) s.reset();
    return s;
}

// Keeps the set, or leaves it to the caller to free.
void give_back(std::unique_ptr<HostStage>& s) {
    if (s->device() >= kDevices) return;
    std::lock_guard<std::mutex> lk(pool().mu);
    auto& d = pool().dev[s->device()];
    if (d.contexts == 0) return;
    for (std::unique_ptr<HostStage>& slot : d.idle)
        if (!slot) {
            slot = std::move(s);
            return;
        }
}

// Whether every copy of the range goes through the driver's own buffers:
// neither page-locked nor managed nor device memory, which it moves directly
// (1920x1080 film into page-locked memory 0.74 ms, through the chunks 3.0; 2^20
// page-locked rays and hits 2.6 and 4.9).
bool pageable(const void* p, size_t bytes) {
    const unsigned char* const ends[2] = {static_cast<const unsigned char*>(p),
                                          static_cast<const unsigned char*>(p) + bytes - 1};
    for (const unsigned char* q : ends) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, q) != cudaSuccess) {
            cudaGetLastError();
            return true;
        }
        if (a.type == cudaMemoryTypeUnregistered) return true;
    }
    return false;
}

cudaError_t staged(void* dst, const void* src, size_t bytes, cudaStream_t st, int device, bool out) {
    if (bytes >= kStageMin && pageable(out ? dst : src, bytes)) {
        if (std::unique_ptr<HostStage> s = take(device)) {
            const cudaError_t e = s->copy(dst, src, bytes, st, out);
            if (e == cudaSuccess) give_back(s);  // after an error its events say nothing: freed
            return e;
        }
    }
    cudaError_t e = cudaMemcpyAsync(dst, src, bytes, out ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && out) e = cudaStreamSynchronize(st);
    return e;
}

}  // namespace

void stage_retain(int device) {
    if (device >= kDevices) return;
    std::lock_guard<std::mutex> lk(pool().mu);
    pool().dev[device].contexts++;
}
void stage_release(int device) {
    if (device >= kDevices) return;
    std::unique_ptr<HostStage> gone[kIdle];  // freed after the lock
    std::lock_guard<std::mutex> lk(pool().mu);
    auto& d = pool().dev[device];
    if (--d.contexts == 0)
        for (int i = 0; i < kIdle; ++i) gone[i] = std::move(d.idle[i]);
}

cudaError_t stage_read(void* dst, const void* src, size_t bytes, cudaStream_t st, int device) {
    return staged(dst, src, bytes, st, device, true);
}
cudaError_t stage_write(void* dst, const void* src, size_t bytes, cudaStream_t st, int device) {
    return staged(dst, src, bytes, st, device, false);
}

}  // namespace ana
