// mem.cu -- where handles get their device memory, streams and page-locked blocks.
//
// A program that builds a matrix or a solver per step (assembly, Galerkin products, a training
// step) made some 60 cudaMalloc / cudaFree / cudaMallocHost calls a step, each mapping or
// unmapping memory and most of them synchronising the device. Device memory comes from one
// pool per device instead, whose allocations are stream-ordered and reuse what was freed; large
// blocks from cudaMalloc, kept in a list of their own; a context's stream and scratch, and the
// page-locked blocks of the solvers' control data, wait in bounded lists for the next handle. All
// of it is safe to use from several threads.
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include "internal.h"

namespace fb {
namespace {

constexpr int kMaxDev = 64;
// Free memory kept for the next handles, 4 GiB a device or about 2% of the card: in the pool
// (checked when a handle or a call's scratch is released: dev_bound) and as large blocks. All of it
// goes back to the device when an allocation of the library fails or the program asks for it
// (fasp_gpu_trim): other allocators of the process do not see it.
constexpr unsigned long long kPoolKeeps = 1ull << 29, kLargeKeeps = 7ull << 29;
// A block of at least kLarge bytes comes from cudaMalloc. The pool maps new memory at some 10 to 20
// ms a GB and unmaps it as slowly, cudaMalloc and cudaFree take 0.7 and 1.4 ms for 1 GB; at 64 MB
// both ways take 0.4 ms (B200). A product with 5 GB of scratch took 137 to 838 ms out of the pool
// (which gave memory back at every wait), 130 to 139 ms this way, and 145 ms before there was a
// pool; one with 24 GB 2,250, 2,050 and 2,070 ms.
constexpr size_t kLarge = (size_t)64 << 20;

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
        unsigned long long keep = ~0ull; // nothing at a synchronisation: see dev_bound
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

// The lists are never destroyed: a handle may outlive the library's static objects.
std::mutex& g_lock = *new std::mutex;
// Idle contexts, and idle page-locked blocks of kPinnedBlock bytes.
constexpr size_t kIdleCtx = 32, kIdlePinned = 64;
std::vector<Ctx>& g_ctx = *new std::vector<Ctx>;
std::vector<void*>& g_pinned = *new std::vector<void*>;

struct Block {
    void*  p;
    size_t bytes;
    int    dev;
};
std::map<void*, Block>& g_large = *new std::map<void*, Block>; // large blocks in use
constexpr size_t kIdleLarge = 64;
Block  g_idle[kIdleLarge];      // and idle ones, oldest first
size_t g_nIdle = 0;

// Takes idle block k out of the list (g_lock held).
Block take_idle(size_t k)
{
    const Block b = g_idle[k];
    for (--g_nIdle; k < g_nIdle; ++k) g_idle[k] = g_idle[k + 1];
    return b;
}

// The smallest idle block of at least `bytes`, at most a quarter larger, or a new one.
cudaError_t large_get(void** p, size_t bytes, int dev)
{
    Block b{nullptr, bytes, dev};
    {
        std::lock_guard<std::mutex> hold(g_lock);
        size_t best = kIdleLarge;
        for (size_t k = 0; k < g_nIdle; ++k)
            if (g_idle[k].dev == dev && g_idle[k].bytes >= bytes &&
                g_idle[k].bytes - bytes <= bytes / 4 &&
                (best == kIdleLarge || g_idle[k].bytes < g_idle[best].bytes))
                best = k;
        if (best < kIdleLarge) b = take_idle(best);
    }
    if (!b.p) {
        const cudaError_t e = cudaMalloc(&b.p, bytes);
        if (e != cudaSuccess) return e;
    }
    *p = b.p;
    try {
        std::lock_guard<std::mutex> hold(g_lock);
        g_large[b.p] = b;
    } catch (const std::bad_alloc&) { // not known as large: dev_free gives it back at once
    }
    return cudaSuccess;
}

// Whether p is a large block: it is idle now, and what is too much of those is given back.
bool large_put(void* p)
{
    Block out[kIdleLarge + 1];
    size_t n = 0;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        const auto it = g_large.find(p);
        if (it == g_large.end()) return false;
        const Block b = it->second;
        g_large.erase(it);
        size_t sum = b.bytes;
        for (size_t k = 0; k < g_nIdle; ++k) sum += g_idle[k].dev == b.dev ? g_idle[k].bytes : 0;
        if (b.bytes > kLargeKeeps) {
            out[n++] = b;
        } else {
            for (size_t k = 0; k < g_nIdle && sum > kLargeKeeps;)
                if (g_idle[k].dev == b.dev) {
                    sum -= g_idle[k].bytes;
                    out[n++] = take_idle(k);
                } else {
                    ++k;
                }
            if (g_nIdle == kIdleLarge) out[n++] = take_idle(0);
            g_idle[g_nIdle++] = b;
        }
    }
    for (size_t k = 0; k < n; ++k) cudaFree(out[k].p);
    return true;
}

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
    Block blocks[kIdleLarge];
    size_t n = 0, nb = 0;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        for (size_t k = g_nIdle; k-- > 0;)
            if (g_idle[k].dev == dev) blocks[nb++] = take_idle(k);
        for (size_t k = g_ctx.size(); k-- > 0;)
            if (g_ctx[k].dev == dev) {
                gone[n++] = g_ctx[k];
                g_ctx.erase(g_ctx.begin() + (ptrdiff_t)k);
            }
    }
    while (n > 0) release(gone[--n]);
    while (nb > 0) cudaFree(blocks[--nb].p);
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
        const cudaError_t e = bytes >= kLarge ? large_get(p, bytes, dev)
                              : pool          ? cudaMallocFromPoolAsync(p, bytes, pool, s)
                                              : cudaMalloc(p, bytes);
        if (e == cudaSuccess) return kOk;
        cudaGetLastError();
        *p = nullptr;
        if (attempt == 0) dev_trim(dev);
    }
    return kErrAlloc;
}

void dev_free(void* p)
{
    if (p && !large_put(p)) cudaFree(p);
}

void dev_bound(int dev)
{
    cudaMemPool_t pool = pool_of(dev);
    unsigned long long reserved = 0, used = 0;
    if (!pool) return;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess ||
        (reserved > used + kPoolKeeps && cudaMemPoolTrimTo(pool, used + kPoolKeeps) != cudaSuccess))
        cudaGetLastError();
}

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
    if (stream) dev_bound(dev); // the handle's arrays are released
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
