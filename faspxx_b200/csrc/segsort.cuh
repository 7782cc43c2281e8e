// segsort.cuh -- device building blocks for constructing CSR matrices: an exclusive scan
// of row counts and a segmented sort of 64-bit keys within row segments (register bitonic
// networks for short rows, a shared-memory bitonic network per segment of up to 4,096
// keys, merge passes above that). Used by the ReadMat conversions (ingest.cu) and the
// sparse matrix product (spgemm.cu). Everything here has internal linkage.
#pragma once

#include <algorithm>
#include <vector>

#include "internal.h"

namespace fb {
namespace {


constexpr int      kScanThreads = 256;
constexpr uint32_t kTile = kScanThreads * 8; // elements per scan tile
constexpr int      kSegMax = 4096;           // keys one block sorts in shared memory
constexpr int      kSegThreads = 512;
constexpr uint64_t kPad = ~0ull;

// Device memory of one conversion on stream s, released when it returns (every conversion
// has waited for its stream by then; a failed one waits here).
struct Tmp {
    cudaStream_t       s;
    std::vector<void*> ptrs;
    explicit Tmp(cudaStream_t st) : s(st) {}
    Tmp(const Tmp&) = delete;
    Tmp& operator=(const Tmp&) = delete;
    ~Tmp()
    {
        cudaStreamSynchronize(s);
        for (void* p : ptrs) dev_free(p);
        int dev = 0;
        cudaGetDevice(&dev);
        dev_bound(dev);
    }
    template <typename T>
    int get(T** p, size_t count)
    {
        const int e = dev_alloc(p, std::max<size_t>(count, 1) * sizeof(T), s);
        if (!e) ptrs.push_back(*p);
        return e;
    }
};

inline int grid_for(size_t work, int block)
{
    return (int)std::max<size_t>(1, std::min<size_t>((work + block - 1) / block, 148 * 16));
}

// ---- exclusive scan of uint32 counts: out[0] = 0, out[i+1] = out[i] + in[i] ----------------

// Exclusive scan of one value per thread across the block; *total gets the block's sum.
__device__ uint32_t block_exclusive(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t ws[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = lane < nw ? ws[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        ws[lane] = s;
    }
    __syncthreads();
    const uint32_t excl = x - v + (wid ? ws[wid - 1] : 0u);
    *total = ws[nw - 1];
    __syncthreads();
    return excl;
}

__global__ void __launch_bounds__(kScanThreads) k_tile_sums(uint32_t n, const uint32_t* __restrict__ in,
                                                             uint32_t* __restrict__ sums)
{
    const size_t base = (size_t)blockIdx.x * kTile + (size_t)threadIdx.x * 8;
    uint32_t s = 0;
    for (int j = 0; j < 8; ++j)
        if (base + j < n) s += in[base + j];
    uint32_t total;
    block_exclusive(s, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One block: exclusive scan of the tile sums in place; out[n] = the grand total.
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t nt, uint32_t* __restrict__ sums,
                                                     uint32_t* __restrict__ outTotal)
{
    uint32_t carry = 0;
    for (size_t c0 = 0; c0 < nt; c0 += (size_t)blockDim.x * 8) {
        const size_t base = c0 + (size_t)threadIdx.x * 8;
        uint32_t v[8], s = 0;
        for (int j = 0; j < 8; ++j) {
            v[j] = base + j < nt ? sums[base + j] : 0u;
            s += v[j];
        }
        uint32_t total;
        uint32_t e = block_exclusive(s, &total) + carry;
        for (int j = 0; j < 8; ++j) {
            if (base + j < nt) sums[base + j] = e;
            e += v[j];
        }
        carry += total;
    }
    if (threadIdx.x == 0) *outTotal = carry;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(uint32_t n, const uint32_t* __restrict__ in,
                                                              const uint32_t* __restrict__ sums,
                                                              uint32_t* __restrict__ out)
{
    const size_t base = (size_t)blockIdx.x * kTile + (size_t)threadIdx.x * 8;
    uint32_t v[8], s = 0;
    for (int j = 0; j < 8; ++j) {
        v[j] = base + j < n ? in[base + j] : 0u;
        s += v[j];
    }
    uint32_t total;
    uint32_t e = block_exclusive(s, &total) + sums[blockIdx.x];
    for (int j = 0; j < 8; ++j) {
        if (base + j < n) out[base + j] = e;
        e += v[j];
    }
}

// out has n + 1 entries; tileSums has ceil(n / kTile) entries. n > 0.
int scan_counts(cudaStream_t s, uint32_t n, const uint32_t* in, uint32_t* out, uint32_t* tileSums)
{
    const uint32_t nt = (uint32_t)((n + (size_t)kTile - 1) / kTile);
    k_tile_sums<<<nt, kScanThreads, 0, s>>>(n, in, tileSums);
    k_scan_sums<<<1, 1024, 0, s>>>(nt, tileSums, out + n);
    k_scan_apply<<<nt, kScanThreads, 0, s>>>(n, in, tileSums, out);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

// ---- row sorts ------------------------------------------------------------------------------

// Rows with lo < length <= G, one group of G lanes per row, bitonic network in registers.
// Every lane of the warp takes part in every shuffle; rows outside the class sort padding.
template <int G>
__global__ void __launch_bounds__(256) k_sort_short(uint32_t nrow, uint32_t lo,
                                                    const uint32_t* __restrict__ rowPtr,
                                                    uint64_t* __restrict__ keys)
{
    const int lane = threadIdx.x % G;
    const size_t groups = (size_t)gridDim.x * blockDim.x / G;
    for (size_t r0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G; r0 < (nrow + groups - 1) / groups * groups;
         r0 += groups) {
        uint32_t b = 0, len = 0;
        if (r0 < nrow) {
            b = rowPtr[r0];
            len = rowPtr[r0 + 1] - b;
        }
        const bool mine = r0 < nrow && len > lo && len <= (uint32_t)G;
        uint64_t v = mine && (uint32_t)lane < len ? keys[b + lane] : kPad;
#pragma unroll
        for (int k = 2; k <= G; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const uint64_t o = __shfl_xor_sync(0xffffffffu, v, j, G);
                const bool keepMin = ((lane & j) == 0) == ((lane & k) == 0);
                v = keepMin ? (o < v ? o : v) : (o > v ? o : v);
            }
        if (mine && (uint32_t)lane < len) keys[b + lane] = v;
    }
}

// One block per segment (start, length <= kSegMax): bitonic network in shared memory.
__global__ void __launch_bounds__(kSegThreads) k_sort_segment(const uint2* __restrict__ segs,
                                                               uint64_t* __restrict__ keys)
{
    __shared__ uint64_t sh[kSegMax];
    const uint2 sg = segs[blockIdx.x];
    uint32_t P = 64;
    while (P < sg.y) P <<= 1;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) sh[i] = i < sg.y ? keys[sg.x + i] : kPad;
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                const uint32_t l = i ^ j;
                if (l > i) {
                    const uint64_t a = sh[i], c = sh[l];
                    if ((a > c) == ((i & k) == 0)) {
                        sh[i] = c;
                        sh[l] = a;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < sg.y; i += blockDim.x) keys[sg.x + i] = sh[i];
}

// Number of keys in a[0, n) below k (a sorted ascending).
__device__ __forceinline__ uint32_t count_below(const uint64_t* a, uint32_t n, uint64_t k)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (a[mid] < k)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// One merge pass over long rows (start, length): sorted runs of w keys are merged in pairs.
// A key's place in the merged pair is its place in its own run plus the number of keys below
// it in the other run (keys are unique, so no two keys compete for a place).
__global__ void k_merge_pass(uint32_t nh, const uint2* __restrict__ rows, uint32_t w,
                             const uint64_t* __restrict__ in, uint64_t* __restrict__ out)
{
    for (uint32_t h = blockIdx.y; h < nh; h += gridDim.y) {
        const uint2 rg = rows[h];
        const uint64_t* src = in + rg.x;
        uint64_t* dst = out + rg.x;
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < rg.y;
             i += (size_t)gridDim.x * blockDim.x) {
            const size_t run = i / w;
            const size_t left = (run & ~(size_t)1) * w;
            const size_t right = left + w;
            const uint64_t k = src[i];
            size_t pos;
            if (right >= rg.y) {
                pos = i; // an unpaired last run stays where it is
            } else if ((run & 1) == 0) {
                const uint32_t rn = (uint32_t)std::min<size_t>(w, rg.y - right);
                pos = i + count_below(src + right, rn, k);
            } else {
                pos = left + (i - right) + count_below(src + left, w, k);
            }
            dst[pos] = k;
        }
    }
}

__global__ void k_copy_rows(uint32_t nh, const uint2* __restrict__ rows,
                            const uint64_t* __restrict__ in, uint64_t* __restrict__ out)
{
    for (uint32_t h = blockIdx.y; h < nh; h += gridDim.y) {
        const uint2 rg = rows[h];
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < rg.y;
             i += (size_t)gridDim.x * blockDim.x)
            out[rg.x + i] = in[rg.x + i];
    }
}

template <typename T>
int stage(Tmp& t, cudaStream_t s, const T* src, size_t count, bool onDevice, const T** out)
{
    if (onDevice) {
        *out = src;
        return kOk;
    }
    T* d = nullptr;
    int e = t.get(&d, count);
    if (e) return e;
    FB_CUDA(cudaMemcpyAsync(d, src, count * sizeof(T), cudaMemcpyHostToDevice, s));
    *out = d;
    return kOk;
}


// What sort_row_keys has to do: rows of 2 to 8 and of 9 to 32 keys, block segments, rows of
// more than kSegMax keys and the longest of those.
struct SortPlan {
    unsigned n8, n32, segs, huge, maxHuge;
};

// Rows by length. With lists: also each segment and each huge row (start, length), in any
// order.
__global__ void __launch_bounds__(256) k_sort_plan(uint32_t nrow, const uint32_t* __restrict__ rowPtr,
                                                   SortPlan* __restrict__ P, uint2* __restrict__ segs,
                                                   uint2* __restrict__ huge)
{
    unsigned n8 = 0, n32 = 0;
    for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrow;
         r += (size_t)gridDim.x * blockDim.x) {
        const uint32_t b = rowPtr[r], len = rowPtr[r + 1] - b;
        if (len <= 1) continue;
        if (len <= 8) {
            ++n8;
        } else if (len <= 32) {
            ++n32;
        } else {
            const unsigned ns = (unsigned)(((size_t)len + kSegMax - 1) / kSegMax);
            const unsigned at = atomicAdd(&P->segs, ns);
            if (segs)
                for (unsigned k = 0; k < ns; ++k) {
                    const uint32_t o = k * (uint32_t)kSegMax;
                    segs[at + k] = make_uint2(b + o, min((uint32_t)kSegMax, len - o));
                }
            if (len > (uint32_t)kSegMax) {
                const unsigned h = atomicAdd(&P->huge, 1u);
                if (huge) huge[h] = make_uint2(b, len);
                atomicMax(&P->maxHuge, len);
            }
        }
    }
    if (__syncthreads_or(n8 != 0) && threadIdx.x == 0) atomicOr(&P->n8, 1u);
    if (__syncthreads_or(n32 != 0) && threadIdx.x == 0) atomicOr(&P->n32, 1u);
}

// Sorts the keys of every row segment [rowPtr[r], rowPtr[r + 1]) ascending (rowPtr on the
// device, 0-based; keys unique within a row, so the order is fully determined).
int sort_row_keys(Ctx& c, Tmp& t, uint32_t nrow, const uint32_t* rowPtr, uint64_t* keys,
                  uint32_t nkeys)
{
    cudaStream_t s = c.stream;
    int e;
    SortPlan* dp = nullptr;
    SortPlan p;
    if ((e = t.get(&dp, 1))) return e;
    const int gp = grid_for(nrow, 256);
    FB_CUDA(cudaMemsetAsync(dp, 0, sizeof(p), s));
    k_sort_plan<<<gp, 256, 0, s>>>(nrow, rowPtr, dp, nullptr, nullptr);
    FB_CUDA(cudaGetLastError());
    FB_CUDA(cudaMemcpyAsync(&p, dp, sizeof(p), cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if (p.n8) k_sort_short<8><<<grid_for((size_t)nrow * 8, 256), 256, 0, s>>>(nrow, 1, rowPtr, keys);
    if (p.n32) k_sort_short<32><<<grid_for((size_t)nrow * 32, 256), 256, 0, s>>>(nrow, 8, rowPtr, keys);
    FB_CUDA(cudaGetLastError());
    if (!p.segs) return kOk;
    uint2 *segs = nullptr, *dh = nullptr;
    if ((e = t.get(&segs, p.segs)) || (e = t.get(&dh, p.huge))) return e;
    FB_CUDA(cudaMemsetAsync(dp, 0, sizeof(p), s));
    k_sort_plan<<<gp, 256, 0, s>>>(nrow, rowPtr, dp, segs, dh);
    for (size_t o = 0; o < p.segs; o += 0x7fffffffu) {
        const size_t cnt = std::min<size_t>(p.segs - o, 0x7fffffffu);
        k_sort_segment<<<(unsigned)cnt, kSegThreads, 0, s>>>(segs + o, keys);
    }
    FB_CUDA(cudaGetLastError());
    if (!p.huge) return kOk;
    uint64_t* alt = nullptr;
    if ((e = t.get(&alt, nkeys))) return e;
    const dim3 g((unsigned)std::min<size_t>((p.maxHuge + 255) / 256, 1024),
                 std::min<uint32_t>(p.huge, 65535));
    uint64_t *src = keys, *dst = alt;
    for (uint64_t w = kSegMax; w < p.maxHuge; w *= 2) {
        k_merge_pass<<<g, 256, 0, s>>>(p.huge, dh, (uint32_t)w, src, dst);
        std::swap(src, dst);
    }
    if (src != keys) k_copy_rows<<<g, 256, 0, s>>>(p.huge, dh, src, keys);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

// ---- rows of up to kRankMost entries in their final order, one pass -------------------------
// An entry on its way into its row: ordered by (column, position in the input).
struct __align__(16) Rec {
    uint32_t col, pos;
    double   val;
};

constexpr uint32_t kRankMost = 128;    // longest row of k_rank_rows: its work grows with len^2
constexpr uint32_t kRankRows = 64;     // rows of a block's turn
constexpr uint32_t kRankEntries = 2048; // entries of a block's turn, in shared memory

// Where k_rank_rows reads entry q: records scattered into their rows, or raw CSR arrays
// (whose columns start at base).
struct RecSource {
    const Rec* rec;
    __device__ __forceinline__ void get(size_t q, uint64_t* key, double* val) const
    {
        const Rec r = rec[q];
        *key = (uint64_t)r.col << 32 | r.pos;
        *val = r.val;
    }
};
struct CsrSource {
    const uint32_t* ci;
    const double*   va;
    const uint32_t* base;
    __device__ __forceinline__ void get(size_t q, uint64_t* key, double* val) const
    {
        *key = (uint64_t)(ci[q] - *base) << 32 | (uint32_t)q;
        *val = va[q];
    }
};

// Row r's entries are inPtr[r] - *base (base null: 0) and on; its place is [outPtr[r],
// outPtr[r + 1]), one longer where miss[r] asks for a 0.0 diagonal (HOLES: the input segment
// has that spare place too, at its end). An entry's place is the number of its row's keys
// below its own (keys are unique), counted in shared memory, plus one past an inserted
// diagonal: no sort, no second pass to insert, no gather of values by position, and all
// global reads and writes of a block are one contiguous range. Bound by the reads of shared
// memory, one key per (entry, entry of its row).
template <bool HOLES, class Source>
__global__ void __launch_bounds__(256) k_rank_rows(uint32_t nrow, const uint32_t* __restrict__ inPtr,
                                                   const uint32_t* __restrict__ base,
                                                   const uint32_t* __restrict__ outPtr,
                                                   const uint8_t* __restrict__ miss, Source src,
                                                   uint32_t* __restrict__ outCol,
                                                   double* __restrict__ outVal)
{
    __shared__ uint64_t key[kRankEntries];
    __shared__ double val[kRankEntries];
    __shared__ uint32_t ib[kRankRows + 1], ob[kRankRows];
    __shared__ uint8_t ms[kRankRows];
    const uint32_t t = threadIdx.x, in0 = base ? *base : 0u;
    const size_t nt = ((size_t)nrow + kRankRows - 1) / kRankRows;
    for (size_t tile = blockIdx.x; tile < nt; tile += gridDim.x) {
        const uint32_t r0 = (uint32_t)(tile * kRankRows);
        const uint32_t rows = nrow - r0 < kRankRows ? nrow - r0 : kRankRows;
        __syncthreads();
        if (t <= rows) ib[t] = inPtr[r0 + t] - in0;
        if (t < rows) {
            ob[t] = outPtr[r0 + t];
            ms[t] = miss ? miss[r0 + t] : (uint8_t)0;
        }
        __syncthreads();
        for (uint32_t s = 0; s < rows;) {
            // as many rows as fit (at least one: a row has at most kRankMost entries and a hole)
            const uint32_t g = (uint32_t)__syncthreads_count(
                t >= s && t < rows && ib[t + 1] - ib[s] <= kRankEntries);
            const uint32_t c0 = ib[s], n = ib[s + g] - c0;
            for (uint32_t q = t; q < n; q += blockDim.x) src.get((size_t)c0 + q, &key[q], &val[q]);
            __syncthreads();
            for (uint32_t q = t; q < n; q += blockDim.x) {
                uint32_t lo = s, hi = s + g; // the row: ib[lo] - c0 <= q < ib[hi] - c0
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) / 2;
                    if (ib[mid] - c0 <= q)
                        lo = mid;
                    else
                        hi = mid;
                }
                const uint32_t b = ib[lo] - c0;
                const uint32_t e = ib[lo + 1] - c0 - (HOLES ? ms[lo] : 0u);
                if (HOLES && q >= e) continue; // the spare place
                const uint64_t k = key[q];
                uint32_t below = 0;
#pragma unroll 4
                for (uint32_t j = b; j < e; ++j) below += key[j] < k ? 1u : 0u;
                const uint32_t col = (uint32_t)(k >> 32);
                const size_t o = (size_t)ob[lo] + below + (ms[lo] && col > r0 + lo ? 1u : 0u);
                outCol[o] = col;
                if (outVal) outVal[o] = val[q];
            }
            if (t >= s && t < s + g && ms[t]) { // the row's explicit 0.0 diagonal
                const uint32_t b = ib[t] - c0, e = ib[t + 1] - c0 - (HOLES ? 1u : 0u);
                uint32_t below = 0;
                for (uint32_t j = b; j < e; ++j) below += (uint32_t)(key[j] >> 32) < r0 + t ? 1u : 0u;
                outCol[(size_t)ob[t] + below] = r0 + t;
                outVal[(size_t)ob[t] + below] = 0.0;
            }
            __syncthreads();
            s += g;
        }
    }
}

template <bool HOLES, class Source>
int rank_rows(Ctx& c, uint32_t nrow, const uint32_t* inPtr, const uint32_t* base,
              const uint32_t* outPtr, const uint8_t* miss, Source src, uint32_t* outCol,
              double* outVal)
{
    const auto kern = k_rank_rows<HOLES, Source>;
    const int g = std::max(1, std::min(ceil_div(nrow, (int)kRankRows),
                                       resident_grid(c, (const void*)kern, 256)));
    kern<<<g, 256, 0, c.stream>>>(nrow, inPtr, base, outPtr, miss, src, outCol, outVal);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

} // namespace
} // namespace fb
