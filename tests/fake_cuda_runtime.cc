// A CUDA runtime of two devices on the host, to be linked with the library's objects in place of
// the real one: kernels do nothing, copies move host memory, and every stream remembers what was
// enqueued on it and what has been waited for. Pool memory given back while its device still has
// work that nobody waited for is counted (the real cudaFree of pool memory does not wait).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace {

struct Stream {
    int           dev;
    unsigned long seq, done;
    bool          capturing;
    std::vector<std::pair<Stream*, unsigned long>> after; // waited for on this stream
};
struct Event {
    Stream*       s;
    unsigned long seq;
};
struct Block {
    size_t bytes;
    int    dev;
    bool   pooled;
};
struct Call {
    dim3         grid, block;
    size_t       smem;
    cudaStream_t stream;
};

constexpr int kDevices = 2;
std::recursive_mutex g_lock;
thread_local int t_dev = 0;
thread_local std::vector<Call> t_calls;
Stream g_legacy[kDevices] = {{0, 0, 0, false, {}}, {1, 0, 0, false, {}}};
std::vector<Stream*> g_streams = {&g_legacy[0], &g_legacy[1]};
std::map<void*, Block> g_blocks;
std::map<const void*, std::string> g_names;
std::vector<std::string> g_launched;
int g_early = 0, g_clusters = 16, g_trims = 0, g_refused = 0;
int g_failIn = -1, g_failures = 0; // device allocations until two in a row fail (a retry with them)
int g_pools[kDevices] = {0, 1};

#define HOLD std::lock_guard<std::recursive_mutex> hold(g_lock)

Stream* of(cudaStream_t s)
{
    return !s || s == cudaStreamLegacy || s == cudaStreamPerThread ? &g_legacy[t_dev] : (Stream*)s;
}
void reached(Stream* s, unsigned long seq)
{
    if (s->done < seq) s->done = seq;
    auto deps = std::move(s->after);
    s->after.clear();
    for (auto& d : deps) reached(d.first, d.second);
}
void idle(int dev)
{
    for (Stream* s : g_streams)
        if (s->dev == dev) reached(s, s->seq);
}
bool busy(int dev)
{
    for (Stream* s : g_streams)
        if (s->dev == dev && s->done < s->seq) return true;
    return false;
}
void enqueue(cudaStream_t st)
{
    Stream* s = of(st);
    if (!s->capturing) ++s->seq;
}
cudaError_t launch(const void* fn, cudaStream_t st)
{
    HOLD;
    g_launched.push_back(g_names.count(fn) ? g_names[fn] : "?");
    enqueue(st);
    return cudaSuccess;
}
cudaError_t allocate(void** p, size_t n, int dev, bool pooled, bool device = true)
{
    HOLD;
    if (device && g_failIn >= 0 && --g_failIn < 0) {
        ++g_failures;
        if (g_failures % 2) g_failIn = 0;
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    *p = std::calloc(n + 256, 1);
    if (!*p) return cudaErrorMemoryAllocation;
    g_blocks[*p] = Block{n, dev, pooled};
    return cudaSuccess;
}

} // namespace

extern "C" {

// ---- what a test sets and reads ----
int  fake_early_frees() { return g_early; }
int  fake_blocks() { return (int)g_blocks.size(); }
void fake_set_clusters(int n) { g_clusters = n; }
void fake_fail_in(int n) { g_failIn = n; }
int  fake_failures() { return g_failures; }
int  fake_refused() { return g_refused; }
int  fake_trims() { return g_trims; }
int  fake_device() { return t_dev; }
void fake_use_device(int dev) { t_dev = dev; }
void* fake_stream() { cudaStream_t s; cudaStreamCreateWithFlags(&s, 0); return s; }
void fake_clear_launches() { g_launched.clear(); }
int  fake_launches(const char* part)
{
    int n = 0;
    for (auto& s : g_launched) n += s.find(part) != std::string::npos;
    return n;
}

// ---- registration ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void   __cudaRegisterFatBinaryEnd(void**) {}
void   __cudaUnregisterFatBinary(void**) {}
void   __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void   __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                              dim3*, dim3*, int*)
{
    g_names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st)
{
    t_calls.push_back(Call{g, b, smem, (cudaStream_t)st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st)
{
    const Call c = t_calls.back();
    t_calls.pop_back();
    *g = c.grid;
    *b = c.block;
    *smem = c.smem;
    *(cudaStream_t*)st = c.stream;
    return cudaSuccess;
}

// ---- devices ----
cudaError_t cudaGetDeviceCount(int* n) { *n = kDevices; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = t_dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d)
{
    if (d < 0 || d >= kDevices) return cudaErrorInvalidDevice;
    t_dev = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { HOLD; idle(t_dev); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n, t_dev, false); }
cudaError_t cudaMallocHost(void** p, size_t n) { return allocate(p, n, t_dev, false, false); }
cudaError_t cudaFreeHost(void* p)
{
    HOLD;
    if (p && g_blocks.erase(p)) std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* pr)
{
    *p = (cudaMemPool_t)&g_pools[pr->location.id];
    return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v)
{
    *(unsigned long long*)v = 0;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { ++g_trims; return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s)
{
    const cudaError_t e = allocate(p, n, *(int*)pool, true);
    if (e == cudaSuccess) enqueue(s);
    return e;
}
cudaError_t cudaFree(void* p)
{
    HOLD;
    if (!p) return cudaSuccess;
    auto it = g_blocks.find(p);
    if (it == g_blocks.end()) return cudaErrorInvalidValue;
    if (!it->second.pooled)
        idle(it->second.dev);
    else if (busy(it->second.dev))
        ++g_early;
    std::free(p);
    g_blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    HOLD;
    std::memcpy(d, s, n);
    enqueue(st);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    HOLD;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
    HOLD;
    std::memset(d, v, n);
    enqueue(st);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, cudaStreamLegacy); }
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind)
{
    std::memset(d, 0, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*)
{
    static char room[1 << 16];
    *p = room;
    return cudaSuccess;
}

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    HOLD;
    Stream* n = new Stream{t_dev, 0, 0, false, {}};
    g_streams.push_back(n);
    *s = (cudaStream_t)n;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    HOLD;
    Stream* s = of(st);
    reached(s, s->seq);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t) new Event{nullptr, 0}; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st)
{
    HOLD;
    *(Event*)e = Event{of(st), of(st)->seq};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    HOLD;
    Event* v = (Event*)e;
    if (v->s) reached(v->s, v->seq);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned)
{
    HOLD;
    Event* v = (Event*)e;
    enqueue(st);
    if (v->s && v->s != of(st)) of(st)->after.push_back({v->s, v->seq});
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
    of(s)->capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g)
{
    of(s)->capturing = false;
    *g = (cudaGraph_t)&g_pools;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long)
{
    *x = (cudaGraphExec_t)&g_pools;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { HOLD; enqueue(s); return cudaSuccess; }

// ---- kernels ----
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) { return launch(f, s); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s)
{
    return launch(f, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**)
{
    for (unsigned k = 0; k < c->numAttrs; ++k)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension && g_clusters == 0) {
            ++g_refused; // no room for a cluster
            return cudaErrorInvalidConfiguration;
        }
    return launch(f, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*)
{
    std::memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*)
{
    *n = g_clusters;
    return cudaSuccess;
}

} // extern "C"
