// A stand-in for the CUDA runtime calls that libfomo_b200.so makes, preloaded
// into a child process so that the library's host code runs without a GPU and
// meets errors on purpose.  Device memory is host memory, kernels are counted
// by name and not run, streams and events are finished at once.
//
// Memory pools keep what they mapped until they are trimmed, and count against
// one capacity, as on a device.  fake_set() makes calls fail or wait.
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <unistd.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
struct Pool {
    size_t used = 0, reserved = 0;
    bool alive = true;
};
struct Block {
    Pool* pool;
    size_t bytes;
};
std::recursive_mutex mu;
std::map<const void*, std::string> kernels;
std::map<std::string, long> launches;
std::map<void*, Block> blocks;
std::map<Pool*, int> pools;
std::map<std::string, long> settings, counts;
thread_local cudaError_t last = cudaSuccess;

long setting(const char* k, long dflt = 0) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    auto it = settings.find(k);
    return it == settings.end() ? dflt : it->second;
}
cudaError_t note(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
size_t capacity() { return (size_t)setting("capacity", 1l << 36); }
size_t reserved() {
    size_t r = 0;
    for (auto& p : pools)
        if (p.first->alive) r += p.first->reserved;
    return r;
}
cudaError_t launch(const void* f) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    launches[kernels[f]] += 1;
    return cudaSuccess;
}
CUresult encode(...) { return setting("fail_encode") ? CUDA_ERROR_INVALID_VALUE : CUDA_SUCCESS; }
// Waits while fake_set("hold", 1): work enqueued on a stream that does not finish yet.
void held() {
    while (setting("hold")) usleep(200);
}
}  // namespace

extern "C" {
void fake_set(const char* k, long v) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    settings[k] = v;
}
// "launches:<part of a kernel's name>", "live_bytes" of pool blocks, "reserved" bytes of live pools,
// "pools" alive, "bad_pool_calls" on a destroyed or null pool
long fake_get(const char* k) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const std::string s = k;
    long n = 0;
    if (s.rfind("launches:", 0) == 0) {
        for (auto& l : launches)
            if (l.first.find(s.substr(9)) != std::string::npos) n += l.second;
        return n;
    }
    if (s == "live_bytes") {
        for (auto& b : blocks) n += b.second.pool ? (long)b.second.bytes : 0;
        return n;
    }
    if (s == "reserved") return (long)reserved();
    if (s == "pools") {
        for (auto& p : pools) n += p.first->alive;
        return n;
    }
    return counts[s];
}

void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    *g = *b = dim3(1);
    *smem = 0;
    *(void**)st = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) { return launch(f); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) {
    const long after = setting("refuse_cooperative_after", -1);
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (after >= 0 && counts["cooperative"] >= after) return note(cudaErrorCooperativeLaunchTooLarge);
    counts["cooperative"] += 1;
    usleep((useconds_t)setting("launch_us"));
    return launch(f);
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->major = 10;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? (int)setting("sm_count", 148) : 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 1, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = (void*)encode;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, note(cudaErrorInvalidSymbol); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    return *x = (cudaGraphExec_t)std::malloc(1), cudaSuccess;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return std::free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return std::free(x), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return setting("hold") ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return held(), cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.01f, cudaSuccess; }

cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    Pool* q = new Pool;
    pools[q] = 1;
    *p = (cudaMemPool_t)q;
    return cudaSuccess;
}
static Pool* live_pool(cudaMemPool_t p) {
    auto it = pools.find((Pool*)p);
    if (it != pools.end() && it->first->alive) return it->first;
    counts["bad_pool_calls"] += 1;
    return nullptr;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    Pool* q = live_pool(p);
    if (!q) return note(cudaErrorInvalidValue);
    q->alive = false;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    Pool* q = live_pool(p);
    if (!q) return note(cudaErrorInvalidValue);
    *(uint64_t*)v = a == cudaMemPoolAttrReservedMemCurrent ? q->reserved : q->used;
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    Pool* q = live_pool(p);
    if (!q) return note(cudaErrorInvalidValue);
    if (q->reserved > keep) q->reserved = keep > q->used ? keep : q->used;
    return cudaSuccess;
}
// fake_set("scale", k): a block counts k times its size in its pool
cudaError_t cudaMallocFromPoolAsync(void** ptr, size_t bytes, cudaMemPool_t p, cudaStream_t) {
    const long lo = setting("fail_alloc_min", -1), hi = setting("fail_alloc_max", -1);
    const size_t n = bytes * (size_t)setting("scale", 1);
    std::lock_guard<std::recursive_mutex> lk(mu);
    Pool* q = live_pool(p);
    if (!q) return note(cudaErrorInvalidValue);
    const size_t grow = q->used + n > q->reserved ? q->used + n - q->reserved : 0;
    const bool asked = lo >= 0 && (long)n >= lo && (long)n <= hi;
    if (asked || reserved() + grow > capacity()) {
        counts["failed_allocs"] += 1;
        return note(cudaErrorMemoryAllocation);
    }
    q->used += n;
    q->reserved += grow;
    blocks[*ptr = std::calloc(bytes ? bytes : 1, 1)] = Block{q, n};
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    auto it = blocks.find(p);
    if (it == blocks.end()) return note(cudaErrorInvalidValue);
    if (it->second.pool) it->second.pool->used -= it->second.bytes;
    blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    blocks[*p = std::calloc(n, 1)] = Block{nullptr, n};
    return cudaSuccess;
}
// fake_set("hold_free", 1): waits, as cudaFree waits for the device ("in_free" counts the calls that did)
cudaError_t cudaFree(void* p) {
    if (setting("hold_free")) {
        {
            std::lock_guard<std::recursive_mutex> lk(mu);
            counts["in_free"] += 1;
        }
        while (setting("hold_free")) usleep(200);
    }
    return cudaFreeAsync(p, nullptr);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::calloc(n ? n : 1, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    *t = capacity();
    *f = *t - reserved();
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memmove(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
}
