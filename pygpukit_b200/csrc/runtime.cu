// runtime.cu -- device memory, streams, events, graph capture and error plumbing of the
// C ABI (include/pgk_b200.h).  Minimal B200 equivalent of the reference's native/core/
// (memory.cpp, stream.cpp, event.cpp, cuda_graph.cpp, device.cpp); no driver-API context
// juggling: one process = one GPU, CUDA runtime primary context.
#include "common.cuh"
#include "tc_common.cuh"
#include "../../include/pgk_b200.h"

#include <atomic>
#include <cstdarg>
#include <cstring>
#include <mutex>

namespace pgk {

static thread_local char g_err[512] = "";
static std::atomic<int64_t> g_launches{0};
static std::atomic<int> g_pdl{0};
static int g_sm_count = 0;

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    // same shape as the reference's "<fn> failed: <cudaGetErrorString>" (error.cuh:28-37)
    const char* base = strrchr(file, '/');
    set_error("%s failed: %s (%s:%d)", what, cudaGetErrorString(e), base ? base + 1 : file, line);
    cudaGetLastError();  // clear sticky-less errors
    return (int)e ? (int)e : 1;
}

// pgk_free() tells interested translation units that an allocation is gone (the FP8 code scanner remembers base
// pointers); registered at load time, so runtime.cu links without them
static void (*g_free_hook)(const void*) = nullptr;
void set_free_hook(void (*fn)(const void*)) { g_free_hook = fn; }

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
bool pdl_enabled() { return g_pdl.load(std::memory_order_relaxed) != 0; }

int sm_count() {
    if (g_sm_count == 0) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0)
            g_sm_count = n;
        else
            g_sm_count = 148;
    }
    return g_sm_count;
}

// ---- stream-ordered work memory: a pool of the library's own per device.  Up to kScratchKeep bytes stay with the pool across
// synchronisations (a fresh mapping costs tens of microseconds); pgk_malloc gives them back when the device runs out.
static const uint64_t kScratchKeep = 256ull << 20;
static std::mutex g_scratch_mu;
static cudaMemPool_t g_scratch[64] = {};

static cudaError_t scratch_pool(cudaMemPool_t* out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    if (!g_scratch[dev]) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // making the pool is no part of a capture
        cudaThreadExchangeStreamCaptureMode(&mode);
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        e = cudaMemPoolCreate(&pool, &props);
        if (e == cudaSuccess) {
            uint64_t keep = kScratchKeep;
            e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return e;
        g_scratch[dev] = pool;
    }
    *out = g_scratch[dev];
    return cudaSuccess;
}

int scratch_alloc(void** ptr, size_t bytes, cudaStream_t st) {
    *ptr = nullptr;
    cudaMemPool_t pool;
    PGK_CUDA(scratch_pool(&pool));
    PGK_CUDA(cudaMallocFromPoolAsync(ptr, bytes ? bytes : 1, pool, st));
    return 0;
}
int scratch_free(void* ptr, cudaStream_t st) {
    if (ptr) PGK_CUDA(cudaFreeAsync(ptr, st));
    return 0;
}
static bool scratch_trim() {
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    bool any = false;
    for (cudaMemPool_t p : g_scratch)
        if (p) any = cudaMemPoolTrimTo(p, 0) == cudaSuccess || any;
    // work memory of captured products whose graphs are gone stays with the device's graph pool, where no other allocation finds it
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) any = cudaDeviceGraphMemTrim(dev) == cudaSuccess || any;
    return any;
}

// ---- staged uploads: the caller's bytes go to a pinned slot and from there in stream order, so that neither side waits for the other.
// (A copy from pageable memory returns once the stream has come to it: a step's description, a few dozen KB, cost the host the whole
// step before, and the device the 130 ... 200 us until the host had launched enough again.)  Eight slots, used by turns; a slot waits
// for its last copy.  Copies above kUploadMax take the plain way and wait.
struct UploadSlot {
    void* host = nullptr;
    size_t bytes = 0;
    cudaEvent_t copied = nullptr;
    int dev = -1;
    bool used = false;                                                  // `copied` has been recorded
};
static constexpr size_t kUploadMax = 1ull << 20;
static constexpr int kUploadSlots = 8;
static UploadSlot g_upload[kUploadSlots];
static int g_upload_next = 0;
static std::mutex g_upload_mu;

static int upload(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    PGK_CUDA(cudaStreamIsCapturing(st, &cs));
    PGK_REQUIRE(cs == cudaStreamCaptureStatusNone, "upload failed: a captured copy would repeat this call's bytes");
    if (bytes > kUploadMax) {
        PGK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        PGK_CUDA(cudaStreamSynchronize(st));
        return wait_check();
    }
    int dev = 0;
    PGK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_upload_mu);
    UploadSlot& s = g_upload[g_upload_next];
    g_upload_next = (g_upload_next + 1) % kUploadSlots;
    if (s.used) PGK_CUDA(cudaEventSynchronize(s.copied));
    s.used = false;
    if (s.bytes < bytes) {
        if (s.host) PGK_CUDA(cudaFreeHost(s.host));
        s.host = nullptr;
        s.bytes = 0;
        size_t n = 64 << 10;
        while (n < bytes) n *= 2;
        PGK_CUDA(cudaHostAlloc(&s.host, n, cudaHostAllocPortable));
        s.bytes = n;
    }
    if (s.dev != dev) {
        if (s.copied) PGK_CUDA(cudaEventDestroy(s.copied));
        s.copied = nullptr;
        s.dev = -1;
        PGK_CUDA(cudaEventCreateWithFlags(&s.copied, cudaEventDisableTiming));
        s.dev = dev;
    }
    memcpy(s.host, src, bytes);
    PGK_CUDA(cudaMemcpyAsync(dst, s.host, bytes, cudaMemcpyHostToDevice, st));
    const cudaError_t e = cudaEventRecord(s.copied, st);
    if (e != cudaSuccess) {                                             // the copy may still read the slot
        cudaStreamSynchronize(st);
        return cuda_fail(e, "cudaEventRecord", __FILE__, __LINE__);
    }
    s.used = true;
    return 0;
}
// slots whose copies are done go back
static void upload_trim() {
    std::lock_guard<std::mutex> lk(g_upload_mu);
    for (UploadSlot& s : g_upload)
        if (s.host && (!s.used || cudaEventQuery(s.copied) == cudaSuccess)) {
            cudaFreeHost(s.host);
            s.host = nullptr;
            s.bytes = 0;
            s.used = false;
        }
}

// ---- bounded waits
static std::mutex g_wait_mu;
static std::atomic<int*> g_wait_words{nullptr};
static std::atomic<int> g_wait_seen[kWaitKinds];

int* wait_word(WaitKind kind) {
    int* w = g_wait_words.load(std::memory_order_acquire);
    if (!w) {
        std::lock_guard<std::mutex> lk(g_wait_mu);
        w = g_wait_words.load(std::memory_order_relaxed);
        if (!w) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // no part of a capture
            cudaThreadExchangeStreamCaptureMode(&mode);
            void* p = nullptr;
            const cudaError_t e = cudaHostAlloc(&p, kWaitKinds * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
            w = (int*)memset(p, 0, kWaitKinds * sizeof(int));
            g_wait_words.store(w, std::memory_order_release);
        }
    }
    return w + kind;
}
int wait_check() {
    static const char* const what[kWaitKinds] = {"gemm_rows", "gemm_fp8_tc", "gemm_fp8_rows", "gemm_nvf4_tc", "seq_attention", "seq_attention_decode", "sdpa_causal_fixed_cache",
                                                  "seq_linear_attention_chunks", "wait_probe"};
    int* w = g_wait_words.load(std::memory_order_acquire);
    if (!w) return 0;
    for (int k = 0; k < kWaitKinds; ++k) {
        if (__atomic_load_n(w + k, __ATOMIC_RELAXED) == 0) continue;
        const int v = __atomic_exchange_n(w + k, 0, __ATOMIC_ACQ_REL);
        if (v == 0) continue;                                               // another thread reports it
        g_wait_seen[k].store(v);
        set_error("%s failed: %s; results since the last synchronisation are not valid", what[k],
                  v == 2 ? "its shared memory is not where it needs it" : "a wait inside its kernel ran out");
        return 1;
    }
    return 0;
}
int wait_raised(WaitKind kind) {
    int* w = g_wait_words.load(std::memory_order_acquire);
    const int now = w ? __atomic_load_n(w + kind, __ATOMIC_ACQUIRE) : 0;
    return now ? now : g_wait_seen[kind].load();
}

__global__ void wait_probe_kernel(int* err, uint32_t limit_ns, int* out) {
    __shared__ __align__(8) uint64_t bar;
    mbar_init(&bar, 1);
    mbar_fence_init();
    *out = bar_wait(err, smem_u32(&bar), 0, limit_ns) ? 1 : 0;              // nobody arrives
}

}  // namespace pgk

using namespace pgk;

static inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

extern "C" {

const char* pgk_last_error(void) { return g_err; }

int pgk_version(void) { return 100; }

int pgk_device_count(int* count) {
    PGK_CUDA(cudaGetDeviceCount(count));
    return 0;
}
int pgk_device_set(int device) {
    PGK_CUDA(cudaSetDevice(device));
    g_sm_count = 0;
    return 0;
}
int pgk_device_get(int* device) {
    PGK_CUDA(cudaGetDevice(device));
    return 0;
}
int pgk_device_props(int device, pgk_device_props_t* out) {
    cudaDeviceProp p;
    PGK_CUDA(cudaGetDeviceProperties(&p, device));
    memset(out, 0, sizeof(*out));
    strncpy(out->name, p.name, sizeof(out->name) - 1);
    out->sm_count = p.multiProcessorCount;
    out->cc_major = p.major;
    out->cc_minor = p.minor;
    out->total_mem = p.totalGlobalMem;
    out->l2_bytes = (size_t)p.l2CacheSize;
    out->max_smem_per_block = (int)p.sharedMemPerBlockOptin;
    return 0;
}
int pgk_sm_count(void) { return sm_count(); }
int pgk_device_sync(void) {
    PGK_CUDA(cudaDeviceSynchronize());
    return wait_check();
}
int pgk_wait_probe(int limit_us, int32_t* ran_out, void* stream) {
    PGK_REQUIRE(limit_us > 0 && limit_us <= 100000, "wait_probe failed: the limit must be 1 ... 100000 us, got %d", limit_us);
    int* err = wait_word(kWaitProbe);
    PGK_REQUIRE(err, "wait_probe failed: no pinned host memory");
    PGK_CUDA(launch(wait_probe_kernel, dim3(1), dim3(1), 0, S(stream), err, 1000u * (uint32_t)limit_us, ran_out));
    return 0;
}
int pgk_mem_info(size_t* free_bytes, size_t* total_bytes) {
    PGK_CUDA(cudaMemGetInfo(free_bytes, total_bytes));
    return 0;
}

int pgk_mem_trim(void) {
    scratch_trim();
    upload_trim();
    cudaGetLastError();
    return 0;
}
int pgk_malloc(void** ptr, size_t bytes) {
    *ptr = nullptr;
    if (bytes == 0) bytes = 1;
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e == cudaErrorMemoryAllocation && scratch_trim()) {       // idle work memory counts as free
        cudaGetLastError();
        e = cudaMalloc(ptr, bytes);
    }
    PGK_CUDA(e);
    return 0;
}
int pgk_free(void* ptr) {
    if (ptr) {
        if (g_free_hook) g_free_hook(ptr);
        PGK_CUDA(cudaFree(ptr));
    }
    return 0;
}
int pgk_host_alloc(void** host_ptr, size_t bytes) {
    PGK_CUDA(cudaHostAlloc(host_ptr, bytes ? bytes : 1, cudaHostAllocDefault));
    return 0;
}
int pgk_host_free(void* host_ptr) {
    if (host_ptr) PGK_CUDA(cudaFreeHost(host_ptr));
    return 0;
}
int pgk_memset(void* ptr, int value, size_t bytes, void* stream) {
    PGK_CUDA(cudaMemsetAsync(ptr, value, bytes, S(stream)));
    return 0;
}
int pgk_memcpy_h2d(void* dst, const void* host_src, size_t bytes, void* stream) {
    PGK_CUDA(cudaMemcpyAsync(dst, host_src, bytes, cudaMemcpyHostToDevice, S(stream)));
    return 0;
}
int pgk_upload(void* dst, const void* host_src, size_t bytes, void* stream) {
    if (bytes == 0) return 0;
    return pgk::upload(dst, host_src, bytes, S(stream));
}
int pgk_memcpy_d2h(void* host_dst, const void* src, size_t bytes, void* stream) {
    PGK_CUDA(cudaMemcpyAsync(host_dst, src, bytes, cudaMemcpyDeviceToHost, S(stream)));
    return 0;
}
int pgk_memcpy_d2d(void* dst, const void* src, size_t bytes, void* stream) {
    PGK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, S(stream)));
    return 0;
}

int pgk_stream_create(void** stream) {
    cudaStream_t s;
    PGK_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    *stream = s;
    return 0;
}
int pgk_stream_destroy(void* stream) {
    PGK_CUDA(cudaStreamDestroy(S(stream)));
    return 0;
}
int pgk_stream_sync(void* stream) {
    PGK_CUDA(cudaStreamSynchronize(S(stream)));
    return wait_check();
}
int pgk_event_create(void** event) {
    cudaEvent_t e;
    PGK_CUDA(cudaEventCreate(&e));
    *event = e;
    return 0;
}
int pgk_event_destroy(void* event) {
    PGK_CUDA(cudaEventDestroy((cudaEvent_t)event));
    return 0;
}
int pgk_event_record(void* event, void* stream) {
    PGK_CUDA(cudaEventRecord((cudaEvent_t)event, S(stream)));
    return 0;
}
int pgk_event_sync(void* event) {
    PGK_CUDA(cudaEventSynchronize((cudaEvent_t)event));
    return wait_check();
}
int pgk_event_elapsed_ms(void* start, void* stop, float* ms) {
    PGK_CUDA(cudaEventElapsedTime(ms, (cudaEvent_t)start, (cudaEvent_t)stop));
    return 0;
}

int pgk_graph_begin(void* stream) {
    PGK_REQUIRE(stream != nullptr, "pgk_graph_begin failed: capture needs a non-default stream");
    PGK_CUDA(cudaStreamBeginCapture(S(stream), cudaStreamCaptureModeThreadLocal));
    return 0;
}
int pgk_stream_capturing(void* stream, int* capturing) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    PGK_CUDA(cudaStreamIsCapturing(S(stream), &cs));
    *capturing = cs != cudaStreamCaptureStatusNone;
    return 0;
}
int pgk_graph_end(void* stream, void** graph_exec) {
    cudaGraph_t g = nullptr;
    PGK_CUDA(cudaStreamEndCapture(S(stream), &g));
    cudaGraphExec_t ge = nullptr;
    cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate", __FILE__, __LINE__);
    *graph_exec = ge;
    return 0;
}
int pgk_graph_launch(void* graph_exec, void* stream) {
    PGK_CUDA(cudaGraphLaunch((cudaGraphExec_t)graph_exec, S(stream)));
    return 0;
}
int pgk_graph_destroy(void* graph_exec) {
    if (graph_exec) PGK_CUDA(cudaGraphExecDestroy((cudaGraphExec_t)graph_exec));
    return 0;
}

int pgk_set_pdl(int enabled) {
    g_pdl.store(enabled ? 1 : 0);
    return 0;
}
int64_t pgk_launch_count(void) { return g_launches.load(); }
void pgk_launch_count_reset(void) { g_launches.store(0); }

static void* g_flush_buf = nullptr;
static const size_t kFlushBytes = 256ull << 20;  // 2x the 126 MB L2
int pgk_flush_l2(void* stream) {
    if (!g_flush_buf) PGK_CUDA(cudaMalloc(&g_flush_buf, kFlushBytes));
    static int v = 0;
    PGK_CUDA(cudaMemsetAsync(g_flush_buf, (v++) & 0xff, kFlushBytes, S(stream)));
    return 0;
}

}  // extern "C"
