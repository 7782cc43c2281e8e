// mem.cu -- where handles get their device memory, streams and page-locked blocks.
//
// A program that builds a matrix or a solver per step (assembly, Galerkin products, a training
// step) made some 60 cudaMalloc / cudaFree / cudaMallocHost calls a step, each mapping or
// unmapping memory and most of them synchronising the device. Device memory comes from one
// pool per device instead, whose allocations are stream-ordered and reuse what was freed; a
// context's stream and scratch, and the page-locked blocks of the solvers' control data, wait
// in bounded lists for the next handle. All of it is safe to use from several threads.
#include <cstring>
#include <mutex>
#include <vector>

#include "internal.h"

namespace fb {
namespace {

constexpr int kMaxDev = 64;
// Free memory that a device's pool keeps: about 2% of the card. The rest goes back to the
// device at the next synchronisation, and all of it when an allocation of the library fails or the
// program asks for it (fasp_gpu_trim): other allocators of the process do not see it.
constexpr unsigned long long kPoolKeeps = 4ull << 30;

struct Pool {
    std::once_flag once;
    cudaMemPool_t  pool = nullptr; // null: the device has none, plain cudaMalloc
};
Pool g_pool[kMaxDev];

cudaMemPool_t pool_of(int dev)
{
    if (dev < 0 || dev >= kMaxDev) return nullptr;
    Pool& P = g_pool[dev];
    std::call_once(P.once, [&] {
        cudaMemPoolProps pr;
        std::memset(&pr, 0, sizeof(pr));
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = dev;
        unsigned long long keep = kPoolKeeps;
        if (cudaMemPoolCreate(&P.pool, &pr) != cudaSuccess) {
            cudaGetLastError();
            P.pool = nullptr;
        } else if (cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep) !=
                   cudaSuccess) {
            cudaGetLastError();
        }
    });
    return P.pool;
}

std::mutex g_lock;
// Idle contexts, and idle page-locked blocks of kPinnedBlock bytes.
constexpr size_t kIdleCtx = 32, kIdlePinned = 64;
std::vector<Ctx> g_ctx;
std::vector<void*> g_pinned;

// What a context that nothing uses any more holds.
void release(Ctx& c)
{
    for (cudaEvent_t& ev : c.joinEv)
        if (ev) cudaEventDestroy(ev);
    dev_free(c.red.partials);
    dev_free(c.red.ticket);
    dev_free(c.dslot);
    pinned_put(c.hslot);
    if (c.ownStream && c.stream) cudaStreamDestroy(c.stream);
    c = Ctx();
}

} // namespace

void device_idle(int dev)
{
    int cur = dev;
    cudaGetDevice(&cur);
    if (cur != dev) cudaSetDevice(dev);
    cudaDeviceSynchronize();
    if (cur != dev) cudaSetDevice(cur);
}

int dev_trim(int dev)
{
    if (dev < 0 || dev >= kMaxDev) return kErrNoDevice;
    device_idle(dev);
    Ctx gone[kIdleCtx]; // their scratch would hold on to whole pieces of the pool
    size_t n = 0;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        for (size_t k = g_ctx.size(); k-- > 0;)
            if (g_ctx[k].dev == dev) {
                gone[n++] = g_ctx[k];
                g_ctx.erase(g_ctx.begin() + (ptrdiff_t)k);
            }
    }
    while (n > 0) release(gone[--n]);
    if (!g_pool[dev].pool || cudaMemPoolTrimTo(g_pool[dev].pool, 0) == cudaSuccess) return kOk;
    cudaGetLastError();
    return kErrCuda;
}

int dev_alloc_bytes(void** p, size_t bytes, cudaStream_t s)
{
    *p = nullptr;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaMemPool_t pool = pool_of(dev);
    for (int attempt = 0; attempt < 2; ++attempt) {
        const cudaError_t e = pool ? cudaMallocFromPoolAsync(p, bytes, pool, s)
                                   : cudaMalloc(p, bytes);
        if (e == cudaSuccess) return kOk;
        cudaGetLastError();
        *p = nullptr;
        if (attempt == 0) dev_trim(dev);
    }
    return kErrAlloc;
}

void dev_free(void* p) { cudaFree(p); }

void* pinned_get()
{
    {
        std::lock_guard<std::mutex> hold(g_lock);
        if (!g_pinned.empty()) {
            void* p = g_pinned.back();
            g_pinned.pop_back();
            std::memset(p, 0, kPinnedBlock);
            return p;
        }
    }
    void* p = nullptr;
    if (cudaMallocHost(&p, kPinnedBlock) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::memset(p, 0, kPinnedBlock);
    return p;
}

void pinned_put(void* p)
{
    if (!p) return;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        if (g_pinned.size() < kIdlePinned) {
            g_pinned.push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

int Ctx::init(int device)
{
    dev = device;
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return kErrNoDevice;
    }
    {
        std::lock_guard<std::mutex> hold(g_lock);
        for (size_t k = g_ctx.size(); k-- > 0;)
            if (g_ctx[k].dev == device) {
                *this = g_ctx[k];
                g_ctx.erase(g_ctx.begin() + (ptrdiff_t)k);
                break;
            }
    }
    if (!stream) {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
        nsm = v > 0 ? v : 148;
        if (nsm * 16 > kMaxGrid) nsm = kMaxGrid / 16;
        FB_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        ownStream = true;
        int e;
        if ((e = dev_alloc(&red.partials, sizeof(double) * kMaxRedValues * kMaxGrid, stream)) ||
            (e = dev_alloc(&red.ticket, sizeof(unsigned) * 4, stream)) ||
            (e = dev_alloc(&dslot, sizeof(double) * kSlots, stream)))
            return e;
        static_assert(sizeof(double) * kSlots <= kPinnedBlock, "slots of one page-locked block");
        if (!(hslot = (double*)pinned_get())) return kErrAlloc;
    }
    // as a new context: counters at zero
    launches = 0;
    FB_CUDA(cudaMemsetAsync(red.ticket, 0, sizeof(unsigned) * 4, stream));
    FB_CUDA(cudaMemsetAsync(dslot, 0, sizeof(double) * kSlots, stream));
    FB_CUDA(cudaStreamSynchronize(stream));
    return kOk;
}

void Ctx::destroy()
{
    if (stream && cudaStreamSynchronize(stream) == cudaSuccess && ownStream && red.partials &&
        red.ticket && dslot && hslot) {
        std::lock_guard<std::mutex> hold(g_lock);
        if (g_ctx.size() < kIdleCtx) {
            g_ctx.push_back(*this);
            *this = Ctx();
            return;
        }
    }
    release(*this);
}

} // namespace fb
