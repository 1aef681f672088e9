// A stand-in for the CUDA runtime and the kernels on the host, so that the host
// side of the library (capi.cpp, prepare.cpp, staging.cpp, film_io.cpp) runs
// without a device: "device" memory is host memory of a chosen capacity, every
// operation completes when it is called, and a test can make calls fail, name
// the kind of a host range, and read what was called.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>

#include "build.h"
#include "kernels.h"

namespace {

struct Range {
    size_t size;
    cudaMemoryType type;
};
std::recursive_mutex g_mu;
std::map<uintptr_t, Range> g_ranges;  // device and page-locked memory, and marked ranges
std::map<std::string, long> g_calls;
std::map<std::string, std::pair<long, long>> g_faults;  // calls to let pass, calls to fail
size_t g_capacity = size_t(1) << 30, g_held = 0, g_largest = 0;
long g_direct_bytes = 0, g_extend_rays = 0, g_bad_records = 0, g_good_records = 0;
thread_local cudaError_t t_last = cudaSuccess;

cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) t_last = e;
    return e;
}
thread_local bool t_own = false;  // in the fake's own bookkeeping

// Counts the call; true when it is to fail.
bool called(const char* fn) {
    struct Own {
        Own() { t_own = true; }
        ~Own() { t_own = false; }
    } own;
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    g_calls[fn]++;
    auto it = g_faults.find(fn);
    if (it == g_faults.end()) return false;
    if (it->second.first > 0) {
        it->second.first--;
        return false;
    }
    if (it->second.second == 0) return false;
    it->second.second--;
    return true;
}
const Range* range_of(const void* p, uintptr_t* base = nullptr) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    auto it = g_ranges.upper_bound(a);
    if (it == g_ranges.begin()) return nullptr;
    --it;
    if (base) *base = it->first;
    return a < it->first + it->second.size ? &it->second : nullptr;
}
template <class T>
T* handle() {
    static std::atomic<uintptr_t> next{1};
    return reinterpret_cast<T*>(next.fetch_add(1));
}

std::atomic<long> g_new{-1};  // allocations to let pass before one fails, -1: none fails

}  // namespace

void* operator new(size_t n) {
    if (!t_own && g_new >= 0 && g_new-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {

// ---- what the tests call --------------------------------------------------
void fake_reset(size_t capacity) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    g_calls.clear();
    g_faults.clear();
    g_capacity = capacity;
    g_largest = 0;
    g_direct_bytes = g_extend_rays = g_bad_records = g_good_records = 0;
}
void fake_fail(const char* fn, long after, long times) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    g_faults[fn] = {after, times};
}
long fake_calls(const char* fn) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    return g_calls[fn];
}
void fake_mark(const void* p, size_t size, int type) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (type < 0) g_ranges.erase(reinterpret_cast<uintptr_t>(p));
    else g_ranges[reinterpret_cast<uintptr_t>(p)] = {size, cudaMemoryType(type)};
}
size_t fake_held() { return g_held; }
size_t fake_largest() { return g_largest; }
long fake_direct_bytes() { return g_direct_bytes; }
long fake_extend_rays() { return g_extend_rays; }
long fake_bad_records() { return g_bad_records; }
long fake_good_records() { return g_good_records; }
void fake_fail_new(long after) { g_new = after; }

// ---- the runtime ----------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) {
    if (called("cudaMalloc")) return ret(cudaErrorMemoryAllocation);
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (n > g_capacity || g_held > g_capacity - n) return ret(cudaErrorMemoryAllocation);
    *p = std::aligned_alloc(256, (n + 255) & ~size_t(255));
    std::memset(*p, 0x5A, n);  // what was there before
    g_ranges[reinterpret_cast<uintptr_t>(*p)] = {n, cudaMemoryTypeDevice};
    g_held += n;
    if (n > g_largest) g_largest = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    called("cudaFree");
    if (!p) return cudaSuccess;
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    auto it = g_ranges.find(reinterpret_cast<uintptr_t>(p));
    if (it == g_ranges.end()) return ret(cudaErrorInvalidValue);
    g_held -= it->second.size;
    g_ranges.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) {
    if (called("cudaHostAlloc")) return ret(cudaErrorMemoryAllocation);
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    *p = std::aligned_alloc(4096, (n + 4095) & ~size_t(4095));
    g_ranges[reinterpret_cast<uintptr_t>(*p)] = {n, cudaMemoryTypeHost};
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    called("cudaFreeHost");
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    g_ranges.erase(reinterpret_cast<uintptr_t>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    called("cudaPointerGetAttributes");
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    std::memset(a, 0, sizeof(*a));
    const Range* r = range_of(p);
    a->type = r ? r->type : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    if (called("cudaMemGetInfo")) return ret(cudaErrorUnknown);
    *t = g_capacity;
    *f = g_capacity > g_held ? g_capacity - g_held : 0;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    if (called("cudaMemcpyAsync")) return ret(cudaErrorUnknown);
    {
        // bytes between the device and memory that is not the library's own
        std::lock_guard<std::recursive_mutex> lk(g_mu);
        const void* host = kind == cudaMemcpyHostToDevice ? s : d;
        const Range* r = range_of(host);
        if (kind != cudaMemcpyDeviceToDevice && (!r || r->type != cudaMemoryTypeHost || n >= (size_t(1) << 20)))
            g_direct_bytes += long(n);
    }
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    called("cudaMemsetAsync");
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset2DAsync(void* d, size_t pitch, int v, size_t w, size_t h, cudaStream_t) {
    called("cudaMemset2DAsync");
    for (size_t y = 0; y < h; ++y) std::memset(static_cast<char*>(d) + y * pitch, v, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) {
    return called("cudaSetDevice") ? ret(cudaErrorInvalidDevice) : cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) {
    if (called("cudaStreamCreateWithFlags")) return ret(cudaErrorUnknown);
    *s = handle<CUstream_st>();
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) {
    called("cudaStreamDestroy");
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    return called("cudaStreamSynchronize") ? ret(cudaErrorUnknown) : cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = handle<CUevent_st>();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    called("cudaEventSynchronize");
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) {
    return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error";
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = t_last;
    t_last = cudaSuccess;
    return e;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = handle<CUgraph_st>();
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = handle<CUgraphExec_st>();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"

// ---- the kernels ----------------------------------------------------------
// Path i of a chunk has an entry at bounce b when i is a multiple
// of b + 1; a film pixel (i, 2 i, 3 i) has weight 2; a ray's hit carries its
// origin's x.
namespace ana {

namespace {
bool walked(uint32_t path, uint32_t bounce) { return path % (bounce + 1) == 0; }
uint32_t entries(uint32_t paths, uint32_t bounce) { return (paths + bounce) / (bounce + 1); }
}  // namespace

DeviceTris::~DeviceTris() {}
int build_tris_on_device(const ana_scene_desc&, uint32_t, cudaStream_t, DeviceTris&, std::string& err) {
    err = "no device build here";
    return ANA_ERR_UNSUPPORTED;
}
void prime_kernels() {}
cudaError_t noalloc_trace_scratch(int, unsigned char** base) {
    static unsigned char* mem = static_cast<unsigned char*>(std::malloc(kNoAllocBytes));
    *base = mem;
    return cudaSuccess;
}
void launch_generate(const Params& p, const LaunchCfg&, cudaStream_t) { p.counters[0] = p.chunk_paths; }
void launch_extend(const Params& p, const LaunchCfg&, cudaStream_t, bool) {
    g_extend_rays += p.counters[p.bounce * kCountersPerBounce];
}
void launch_shade(const Params& p, const LaunchCfg&, cudaStream_t) {
    if (p.bounce < p.S.scenes[0].max_depth)
        p.counters[(p.bounce + 1) * kCountersPerBounce] = entries(p.chunk_paths, p.bounce + 1);
}
void launch_shadow(const Params&, const LaunchCfg&, cudaStream_t) {}
void launch_mis(const Params&, const LaunchCfg&, cudaStream_t) {}
void launch_adj_init(const Params&, const LaunchCfg&, cudaStream_t) {}
void launch_keep_hits(const Params& p, const LaunchCfg&, cudaStream_t) {
    for (uint32_t i = 0; i < p.chunk_paths; ++i)
        if (walked(i, p.bounce)) p.a.kept[p.bounce * p.a.kept_stride + i] = make_float4(1.f, 0.f, 0.f, 0.f);
}
// Every path's record of the bounce is a hit of this chunk, or says that the
// path was not there.
void launch_shade_adj(const Params& p, const LaunchCfg& c, cudaStream_t s) {
    if (p.a.kept)
        for (uint32_t i = 0; i < p.chunk_paths; ++i) {
            const float4 h = p.a.kept[p.bounce * p.a.kept_stride + i];
            uint32_t prim;
            std::memcpy(&prim, &h.y, 4);
            ++(prim == (walked(i, p.bounce) ? 0u : 0xFEFEFEFEu) ? g_good_records : g_bad_records);
            p.a.kept[p.bounce * p.a.kept_stride + i].y = 3e33f;  // the next chunk's must be written again
        }
    launch_shade(p, c, s);
}
void launch_shadow_adj(const Params&, const LaunchCfg&, cudaStream_t) {}
void launch_mis_adj(const Params&, const LaunchCfg&, cudaStream_t) {}
void launch_adj_direct(const Params&, const LaunchCfg&, cudaStream_t) {}
void launch_film(const Params& p, const LaunchCfg&, cudaStream_t) {
    for (uint32_t q = 0; q < p.chunk_pixels; ++q) {
        const uint32_t i = q + p.segs[0].first_pixel;  // one scene, one run a chunk
        p.film[i] = ana_film_pixel{float(i), 2.f * float(i), 3.f * float(i), 2.f, 0.f};
        if (p.aov) {
            const float a[8] = {float(i), 1.f, 2.f, 4.f, 3.f, float(i), 5.f, 0.f};
            std::memcpy(p.aov + 8 * size_t(i), a, sizeof(a));
        }
    }
}
void launch_film_image(const ana_film_pixel* film, uint32_t n, float* out, cudaStream_t) {
    for (size_t i = 0; i < n; ++i) {
        const ana_film_pixel& f = film[i];
        out[3 * i] = f.w > 0.f ? f.r / f.w : 0.f;
        out[3 * i + 1] = f.w > 0.f ? f.g / f.w : 0.f;
        out[3 * i + 2] = f.w > 0.f ? f.b / f.w : 0.f;
    }
}
void launch_aov_image(const float* aov, uint32_t n, int layer, float* out, cudaStream_t) {
    for (size_t i = 0; i < n; ++i) {
        const float* a = aov + 8 * i + 4 * layer;
        const float inv = a[3] > 0.f ? 1.f / a[3] : 0.f;
        for (int k = 0; k < 3; ++k) out[3 * i + k] = a[3] > 0.f ? a[k] * inv : 0.f;
    }
}
void launch_trace_batch(const DevScene&, uint32_t, const float* rays, const float* times, size_t n, ana_hit* out, int,
                        uint32_t*, uint32_t*, int, cudaStream_t) {
    for (size_t i = 0; i < n; ++i)
        out[i] = ana_hit{1, 0, int32_t(i & 0xFFFF), -1, rays[8 * i], times ? times[i] : 0.f, 0.f, 0.f};
}
void launch_bsdf_query(const DevMaterial&, const ana_bsdf_query*, uint32_t n, ana_bsdf_result* out, cudaStream_t) {
    std::memset(out, 0, n * sizeof(*out));
}

}  // namespace ana
