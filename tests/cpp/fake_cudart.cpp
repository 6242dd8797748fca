// A stand-in for the CUDA runtime, linked with the library's object files for
// tests of its host code on a machine without a GPU: device memory is host
// memory of a bounded size, streams and events are handles, a kernel launch
// records the kernel's name and runs nothing. A test can make the next
// launches or pool allocations fail and can set how much memory is left.
//
// Memory of a stream-ordered pool follows the documented rules at their
// strictest: what is freed on a stream stays reserved until the stream has been
// synchronised and the pool is trimmed after that.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

constexpr size_t kUnlimited = SIZE_MAX / 2;

struct Fake {
    std::map<const void *, std::string> kernels;
    std::string log;                     // launched kernels' names, one per line
    long fail_launch = -1, fail_pool = -1;   // countdown to the failing call(s)
    bool fail_pool_all = false;          // every pool allocation from then on
    size_t capacity = kUnlimited, used = 0;
    std::map<void *, size_t> blocks, pool_live, pool_pending, pool_ready;
    size_t pool_reserved = 0;
    int capturing = 0;
    size_t synced_log = 0;               // length of the log at the last synchronisation
    int optin = 232448;                  // shared memory a block may opt in to
    cudaError_t last = cudaSuccess;
};

Fake &f()
{
    static Fake *x = new Fake;
    return *x;
}

cudaError_t ret(cudaError_t e)
{
    if (e != cudaSuccess) f().last = e;
    return e;
}

bool countdown(long &n)
{
    if (n < 0) return false;
    return n-- == 0;
}

size_t left()
{
    const size_t held = f().used + f().pool_reserved;
    return held < f().capacity ? f().capacity - held : 0;
}

void synced()
{
    f().synced_log = f().log.size();
    for (auto &b : f().pool_pending) f().pool_ready.insert(b);
    f().pool_pending.clear();
}

cudaError_t launch(const void *fn, void **args)
{
    if (countdown(f().fail_launch)) return ret(cudaErrorLaunchOutOfResources);
    const auto k = f().kernels.find(fn);
    const std::string name = k == f().kernels.end() ? std::string("?") : k->second;
    f().log += name + "\n";
    // the one result that the host code goes on: k_rows_mrange(Space, tables, r0,
    // r1, out), answered with the whole (N-2)-space (Space's seventh word)
    if (name.find("k_rows_mrange") != std::string::npos) {
        uint32_t *out = *static_cast<uint32_t **>(args[4]);
        out[0] = 0;
        out[1] = static_cast<const uint32_t *>(args[0])[6] - 1;
    }
    return cudaSuccess;
}

struct Config {
    dim3 grid, block;
    size_t smem;
    void *stream;
};
thread_local std::vector<Config> t_configs;

}  // namespace

#define API extern "C" __attribute__((visibility("default")))

// ---- the test's side --------------------------------------------------------
API void fake_reset()
{
    f().log.clear();
    f().fail_launch = f().fail_pool = -1;
    f().fail_pool_all = false;
    f().capacity = kUnlimited;
    f().capturing = 0;
    f().optin = 232448;
    f().last = cudaSuccess;
}
API const char *fake_log() { return f().log.c_str(); }
API void fake_clear_log()
{
    f().log.clear();
    f().synced_log = 0;
}
API size_t fake_synced_log() { return f().synced_log; }
API void fake_capture(int on) { f().capturing = on; }
API void fake_fail_launch(long k) { f().fail_launch = k; }
API void fake_fail_pool(long k, int all)
{
    f().fail_pool = k;
    f().fail_pool_all = all != 0;
}
// Leaves this many bytes beside everything that is allocated or held by a pool now.
API void fake_headroom(size_t bytes) { f().capacity = f().used + f().pool_reserved + bytes; }
API size_t fake_pool_held() { return f().pool_reserved; }
API size_t fake_used() { return f().used; }
API void fake_optin(int bytes) { f().optin = bytes; }

// ---- memory -----------------------------------------------------------------
API cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = nullptr;
    if (n > left()) return ret(cudaErrorMemoryAllocation);
    *p = std::calloc(1, n ? n : 1);
    if (!*p) return ret(cudaErrorMemoryAllocation);
    f().blocks[*p] = n;
    f().used += n;
    return cudaSuccess;
}
API cudaError_t cudaFree(void *p)
{
    const auto b = f().blocks.find(p);
    if (b != f().blocks.end()) {
        f().used -= b->second;
        f().blocks.erase(b);
        std::free(p);
    }
    return cudaSuccess;
}
API cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *)
{
    *p = reinterpret_cast<cudaMemPool_t>(0x1000);
    return cudaSuccess;
}
API cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
API cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr a, void *v)
{
    if (a != cudaMemPoolAttrReservedMemCurrent) return ret(cudaErrorInvalidValue);
    *static_cast<uint64_t *>(v) = f().pool_reserved;
    return cudaSuccess;
}
API cudaError_t cudaMemGetInfo(size_t *free, size_t *total)
{
    *free = left();
    *total = f().capacity;
    return cudaSuccess;
}
API cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t)
{
    for (auto &b : f().pool_ready) {
        f().pool_reserved -= b.second;
        std::free(b.first);
    }
    f().pool_ready.clear();
    return cudaSuccess;
}
API cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t)
{
    *p = nullptr;
    if (f().fail_pool == 0) {
        if (!f().fail_pool_all) f().fail_pool = -1;
        return ret(cudaErrorMemoryAllocation);
    }
    if (f().fail_pool > 0) --f().fail_pool;
    for (auto *m : {&f().pool_ready, &f().pool_pending})   // same stream: reused at once
        for (auto b = m->begin(); b != m->end(); ++b)
            if (b->second == n) {
                *p = b->first;
                f().pool_live[*p] = n;
                m->erase(b);
                return cudaSuccess;
            }
    if (n > left()) return ret(cudaErrorMemoryAllocation);
    *p = std::calloc(1, n);
    f().pool_live[*p] = n;
    f().pool_reserved += n;
    return cudaSuccess;
}
API cudaError_t cudaFreeAsync(void *p, cudaStream_t)
{
    const auto b = f().pool_live.find(p);
    if (b == f().pool_live.end()) return ret(cudaErrorInvalidValue);
    f().pool_pending.insert(*b);
    f().pool_live.erase(b);
    return cudaSuccess;
}
API cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
API cudaError_t cudaMemset(void *d, int v, size_t n)
{
    std::memset(d, v, n);
    return cudaSuccess;
}
API cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
    std::memset(d, v, n);
    return cudaSuccess;
}
API cudaError_t cudaGetSymbolAddress(void **p, const void *)
{
    static void *array = std::calloc(1, 64 << 20);
    *p = array;
    return cudaSuccess;
}

// ---- launches -----------------------------------------------------------------
API cudaError_t cudaLaunchKernel(const void *fn, dim3, dim3, void **args, size_t, cudaStream_t)
{
    return launch(fn, args);
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *fn, void **args) { return launch(fn, args); }
API cudaError_t cudaLaunchCooperativeKernel(const void *fn, dim3, dim3, void **args, size_t, cudaStream_t)
{
    return launch(fn, args);
}
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *st)
{
    t_configs.push_back({g, b, smem, st});
    return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st)
{
    if (t_configs.empty()) return cudaErrorMissingConfiguration;
    const Config c = t_configs.back();
    t_configs.pop_back();
    *g = c.grid;
    *b = c.block;
    *smem = c.smem;
    *static_cast<void **>(st) = c.stream;
    return cudaSuccess;
}
API void **__cudaRegisterFatBinary(void *)
{
    static void *handle = nullptr;
    return &handle;
}
API void __cudaRegisterFatBinaryEnd(void **) {}
API void __cudaUnregisterFatBinary(void **) {}
API void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *,
                                dim3 *, int *)
{
    f().kernels[host] = name;
}
API void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
API cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
API cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *)
{
    std::memset(a, 0, sizeof *a);
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t)
{
    *n = 1;
    return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}

// ---- device, streams, events, graphs --------------------------------------------
API cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return cudaSuccess;
}
API cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
API cudaError_t cudaSetDevice(int) { return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount               ? 148
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin    ? f().optin
         : a == cudaDevAttrComputeCapabilityMajor          ? 10
         : a == cudaDevAttrComputeCapabilityMinor          ? 0
                                                           : 1;
    return cudaSuccess;
}
API cudaError_t cudaDeviceSynchronize()
{
    synced();
    return cudaSuccess;
}
API const char *cudaGetErrorString(cudaError_t e)
{
    return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaSuccess ? "no error" : "fake error";
}
API cudaError_t cudaGetLastError()
{
    const cudaError_t e = f().last;
    f().last = cudaSuccess;
    return e;
}
API cudaError_t cudaPeekAtLastError() { return f().last; }
static cudaError_t handle(void **h)
{
    static uintptr_t next = 0x2000;
    *h = reinterpret_cast<void *>(next += 16);
    return cudaSuccess;
}
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle((void **)s); }
API cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    synced();
    return cudaSuccess;
}
API cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
API cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s)
{
    *s = f().capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
API cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    f().capturing = 1;
    return cudaSuccess;
}
API cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    f().capturing = 0;
    return handle((void **)g);
}
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) { return handle((void **)g); }
API cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
API cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle((void **)e); }
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle((void **)e); }
API cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaEventSynchronize(cudaEvent_t)
{
    synced();
    return cudaSuccess;
}
API cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.0f;
    return cudaSuccess;
}
