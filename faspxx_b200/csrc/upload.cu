// upload.cu -- building a Mat in device memory: the structure check (CheckCSR), the diagonal
// (FormDiagPtr, GetDiag), the facts the kernels' dispatch reads (longest row, tile span, one
// diagonal value, 16-bit reach) and the row-class and stencil-mask forms, all computed on the
// device from the arrays in device memory.
#include <algorithm>
#include <cstring>
#include <map>
#include <vector>

#include "internal.h"

namespace fb {

// 32 spare bytes keep vectorised/bulk tail accesses inside the allocation (the warp
// tiles' 16-byte loads read up to 3 entries past the last one)
int dmalloc(void** p, size_t bytes, cudaStream_t s) { return dev_alloc_bytes(p, bytes + 32, s); }

namespace {

// ---- one pass over the structure -----------------------------------------------------------

constexpr uint32_t kRcMaxClasses = 4096;
constexpr uint32_t kRcMaxRowLen = 64;
constexpr uint32_t kRcSlots = 16384; // hash slots: at most a quarter used
constexpr uint32_t kRcProbes = 64;
constexpr uint32_t kRcSample = 8192; // rows looked at first: twice the classes allowed

// What the inspection and the class pass report to the host.
struct Inspect {
    unsigned           bad;     // CheckCSR fails
    unsigned           maxLen;  // longest row
    unsigned           span[6]; // most entries of a tile of 256 >> k rows, widened to multiples of 4
    unsigned           far16;   // some entry is more than 32,767 columns from its row
    unsigned           noDiag;  // some row stores no diagonal entry
    unsigned           classes; // distinct rows met by the class pass
    unsigned           rcStop;  // the rows do not fit the class form
    unsigned           entries; // entries of the class table
    unsigned long long dmin, dmax; // least and greatest diagonal value, as bit patterns
};

constexpr uint32_t kInspectChunk = 4096;
constexpr uint32_t kInspectLong = 128; // longer rows are scanned by the whole block

// A block takes 256 consecutive rows, whose entries are one contiguous range; it copies the
// columns through shared memory in coalesced chunks and each thread scans its own row's part
// (thread per row straight from global memory reads words 4 len bytes apart). A long row's part is
// scanned by all threads: left to its own thread, 64 rows of 500,000 entries took 550 ms. No column is
// trusted: a row whose pointers are not 0 <= b <= e <= nnz is flagged and left out, and
// nothing is indexed by a column here. Bound by the 4 nnz bytes of the columns, 12 n of
// diagonal written and 8 n of diagonal values gathered.
__global__ void __launch_bounds__(kBlock) k_inspect(uint32_t nrow, uint32_t mcol, uint32_t nnz,
                                                    const uint32_t* __restrict__ rowPtr,
                                                    const uint32_t* __restrict__ colInd,
                                                    const double* __restrict__ val,
                                                    uint32_t* __restrict__ diagPtr,
                                                    double* __restrict__ diag,
                                                    Inspect* __restrict__ out)
{
    __shared__ uint32_t cs[kInspectChunk];
    // the tile's long rows in order: begin, end, row, first position of the diagonal
    __shared__ uint32_t lb[kTileRows], le[kTileRows], lr[kTileRows], lp[kTileRows];
    __shared__ uint32_t warpLong[kTileRows / 32];
    bool bad = false, far = false, noDiag = false;
    unsigned maxLen = 0, span[6] = {};
    unsigned long long dmin = ~0ull, dmax = 0ull;
    const size_t ntiles = ((size_t)nrow + kTileRows - 1) / kTileRows;
    for (size_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const size_t t0 = t * kTileRows, row = t0 + threadIdx.x;
        const size_t t1 = t0 + kTileRows < nrow ? t0 + kTileRows : nrow;
        const uint32_t T0 = rowPtr[t0];
        uint32_t T1 = rowPtr[t1], b = 0, e = 0;
        const bool in = row < nrow;
        if (in) {
            b = rowPtr[row];
            e = rowPtr[row + 1];
            if (b > e || e > nnz || (row == 0 && b != 0) || (row + 1 == nrow && e != nnz)) {
                bad = true;
                b = e = 0;
            }
        }
        if (T0 > T1 || T1 > nnz) T1 = T0; // a row of the tile is flagged: nothing to scan
#pragma unroll
        for (int k = 0; k < 6; ++k) // the tile's parts of 256 >> k rows that begin at this row
            if (in && (threadIdx.x & ((kTileRows >> k) - 1)) == 0) {
                const size_t r1 = row + (kTileRows >> k) < t1 ? row + (kTileRows >> k) : t1;
                const uint32_t p0 = rowPtr[row], p1 = rowPtr[r1];
                const unsigned long long w =
                    p1 < p0 ? 0ull : (((unsigned long long)p1 + 3) & ~3ull) - (p0 & ~3u);
                span[k] = max(span[k], (unsigned)(w < 0xffffffffull ? w : 0xffffffffull));
            }
        maxLen = max(maxLen, e - b);
        bool found = false;
        uint32_t dp = 0, nlong = 0, mine = 0, cur = 0;
        const bool isLong = e - b > kInspectLong;
        if (__syncthreads_or(isLong)) {
            const uint32_t bal = __ballot_sync(0xffffffffu, isLong);
            if ((threadIdx.x & 31) == 0) warpLong[threadIdx.x >> 5] = (uint32_t)__popc(bal);
            __syncthreads();
            for (uint32_t w = 0; w < kTileRows / 32; ++w) {
                if (w == threadIdx.x >> 5) mine = nlong;
                nlong += warpLong[w];
            }
            mine += (uint32_t)__popc(bal & ((1u << (threadIdx.x & 31)) - 1u));
            if (isLong) {
                lb[mine] = b;
                le[mine] = e;
                lr[mine] = (uint32_t)row;
                lp[mine] = 0xffffffffu;
            }
        }
        for (size_t c0 = T0; c0 < T1; c0 += kInspectChunk) {
            const uint32_t len = (uint32_t)(T1 - c0 < kInspectChunk ? T1 - c0 : kInspectChunk);
            __syncthreads(); // the previous chunk is done with
            for (uint32_t k = threadIdx.x; k < len; k += kBlock) cs[k] = ld_stream(colInd + c0 + k);
            __syncthreads();
            while (cur < nlong && le[cur] <= c0) ++cur;
            for (uint32_t l = cur; l < nlong && lb[l] < c0 + len; ++l) {
                const size_t lo = lb[l] > c0 ? lb[l] : c0, hi = le[l] < c0 + len ? le[l] : c0 + len;
                const long long r = lr[l];
                for (size_t k = lo + threadIdx.x; k < hi; k += kBlock) {
                    const uint32_t c = cs[k - c0];
                    const long long d = (long long)c - r;
                    bad = bad || c >= mcol;
                    far = far || d < -32767 || d > 32767;
                    if (d == 0) atomicMin(&lp[l], (uint32_t)k);
                }
            }
            const size_t lo = b > c0 ? b : c0, hi = isLong ? lo : e < c0 + len ? e : c0 + len;
            for (size_t k = lo; k < hi; ++k) {
                const uint32_t c = cs[k - c0];
                const long long d = (long long)c - (long long)row;
                bad = bad || c >= mcol;
                far = far || d < -32767 || d > 32767;
                if (d == 0 && !found) {
                    found = true;
                    dp = (uint32_t)k;
                }
            }
        }
        if (nlong) {
            __syncthreads(); // every long row is scanned
            if (isLong && lp[mine] != 0xffffffffu) {
                found = true;
                dp = lp[mine];
            }
        }
        if (in) {
            // FormDiagPtr (MAT.cxx:917-928): the first position whose column is the row, 0
            // where there is none; GetDiag (MAT.cxx:256-267) reads the values there
            diagPtr[row] = dp;
            const double dv = val ? val[dp] : 1.0;
            diag[row] = dv;
            if (found) {
                const unsigned long long bits = (unsigned long long)__double_as_longlong(dv);
                dmin = min(dmin, bits);
                dmax = max(dmax, bits);
            } else {
                noDiag = true;
            }
        }
    }
    const bool anyBad = __syncthreads_or(bad), anyFar = __syncthreads_or(far),
               anyNoDiag = __syncthreads_or(noDiag);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        maxLen = max(maxLen, __shfl_down_sync(0xffffffffu, maxLen, o));
#pragma unroll
        for (int k = 0; k < 6; ++k) span[k] = max(span[k], __shfl_down_sync(0xffffffffu, span[k], o));
        dmin = min(dmin, __shfl_down_sync(0xffffffffu, dmin, o));
        dmax = max(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
    }
    if (threadIdx.x == 0) {
        if (anyBad) atomicOr(&out->bad, 1u);
        if (anyFar) atomicOr(&out->far16, 1u);
        if (anyNoDiag) atomicOr(&out->noDiag, 1u);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out->maxLen, maxLen);
#pragma unroll
        for (int k = 0; k < 6; ++k) atomicMax(&out->span[k], span[k]);
        atomicMin(&out->dmin, dmin);
        atomicMax(&out->dmax, dmax);
    }
}

// ---- row classes ------------------------------------------------------------------------
// A row's class is its length, its column offsets col - row and its values (bit patterns),
// in CSR order. Constant-coefficient stencil matrices have a handful of classes (interior,
// faces, edges, corners), so the SpMV streams a 2-byte class id per row instead of 8 to 12
// bytes per entry. The table is built only when it stays small against the matrix.
//
// k_class_hash puts every row's 64-bit hash into an open-addressed table (key, least row that
// has it) and notes the row's slot; k_class_table sorts the classes by their first row and
// copies their offsets and values; k_class_assign turns slots into class ids and compares
// every row with its class's table entries, so two rows that share a hash but differ are
// found (the pass is then repeated with another seed). The pass goes over kRcSample rows
// spread over the matrix first: one with a coefficient per cell is found unfit there. Left to
// the whole grid, its first wave of 300,000 threads filled the table and all probed it to the
// limit before the stop flag reached them (248 us at 250,000 rows, 13 us with the sample).

struct ClassSlots {
    unsigned long long key[kRcSlots]; // 0: free
    unsigned           rep[kRcSlots]; // least row of the class
};

__global__ void __launch_bounds__(kBlock) k_class_hash(uint32_t nrow, uint32_t step, uint32_t nnz,
                                                       const uint32_t* __restrict__ rowPtr,
                                                       const uint32_t* __restrict__ colInd,
                                                       const double* __restrict__ val,
                                                       unsigned long long seed,
                                                       ClassSlots* __restrict__ S,
                                                       uint16_t* __restrict__ slot,
                                                       Inspect* __restrict__ out)
{
    volatile unsigned* stop = &out->rcStop;
    for (size_t row = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * step; row < nrow;
         row += (size_t)gridDim.x * blockDim.x * step) {
        if (*stop) return;
        const uint32_t b = rowPtr[row], e = rowPtr[row + 1];
        if (b > e || e > nnz || e - b > kRcMaxRowLen) { // not CSR (reported), or too long
            *stop = 1u;
            return;
        }
        unsigned long long h = seed ^ (e - b);
        for (uint32_t k = b; k < e; ++k) {
            const unsigned long long d = (unsigned long long)((long long)colInd[k] - (long long)row);
            h = (h ^ d) * 1099511628211ull;
            h = (h ^ (unsigned long long)__double_as_longlong(val[k])) * 1099511628211ull;
            h ^= h >> 29; // the slot index comes from the low bits
        }
        if (h == 0) h = 1;
        uint32_t s = (uint32_t)(h >> 7) & (kRcSlots - 1), probe = 0;
        for (;; s = (s + 1) & (kRcSlots - 1)) {
            // a copy in L1 may be old: only its answer "this class" counts
            unsigned long long key;
            asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(key) : "l"(&S->key[s]) : "memory");
            if (key != h) key = *(volatile unsigned long long*)&S->key[s];
            if (key == 0) {
                key = atomicCAS(&S->key[s], 0ull, h);
                if (key == 0) {
                    if (atomicAdd(&out->classes, 1u) >= kRcMaxClasses) *stop = 1u;
                    key = h;
                }
            }
            if (key == h) break;
            if (++probe >= kRcProbes || *stop) {
                *stop = 1u;
                return;
            }
        }
        // most rows find a smaller row there already (a copy in L1 is never too small): no atomic
        unsigned rep;
        asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(rep) : "l"(&S->rep[s]) : "memory");
        if (rep > (unsigned)row) atomicMin(&S->rep[s], (unsigned)row);
        slot[row] = (uint16_t)s;
    }
}

// One block: the classes in the order of their first rows, their offsets into the table, and
// the table itself (at most maxEntries entries; more stops the form).
__global__ void __launch_bounds__(1024) k_class_table(const uint32_t* __restrict__ rowPtr,
                                                      const uint32_t* __restrict__ colInd,
                                                      const double* __restrict__ val,
                                                      const ClassSlots* __restrict__ S,
                                                      uint32_t maxEntries,
                                                      uint16_t* __restrict__ idOf,
                                                      uint32_t* __restrict__ off,
                                                      int32_t* __restrict__ delta,
                                                      double* __restrict__ tval,
                                                      Inspect* __restrict__ out)
{
    __shared__ unsigned long long key[kRcMaxClasses]; // first row << 14 | slot
    __shared__ uint32_t cnt, total;
    static_assert(kRcSlots == 1u << 14, "slot bits of the sort key");
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < kRcSlots; s += blockDim.x)
        if (S->key[s]) {
            const uint32_t i = atomicAdd(&cnt, 1u);
            if (i < kRcMaxClasses) key[i] = (unsigned long long)S->rep[s] << 14 | s;
        }
    __syncthreads();
    const uint32_t C = cnt < kRcMaxClasses ? cnt : kRcMaxClasses;
    uint32_t P = 2;
    while (P < C) P <<= 1;
    for (uint32_t i = C + threadIdx.x; i < P; i += blockDim.x) key[i] = ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                const uint32_t l = i ^ j;
                if (l > i) {
                    const unsigned long long a = key[i], c = key[l];
                    if ((a > c) == ((i & k) == 0)) {
                        key[i] = c;
                        key[l] = a;
                    }
                }
            }
            __syncthreads();
        }
    // offsets: one warp, 32 classes at a time
    if (threadIdx.x < 32) {
        uint32_t carry = 0;
        for (uint32_t c0 = 0; c0 < C; c0 += 32) {
            const uint32_t i = c0 + threadIdx.x;
            uint32_t len = 0;
            if (i < C) {
                const uint32_t r = (uint32_t)(key[i] >> 14);
                len = rowPtr[r + 1] - rowPtr[r];
                idOf[key[i] & (kRcSlots - 1)] = (uint16_t)i;
            }
            uint32_t x = len;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)threadIdx.x >= o) x += y;
            }
            if (i < C) off[i] = carry + x - len;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (threadIdx.x == 0) {
            off[C] = carry;
            total = carry;
            out->entries = carry;
            if (carry > maxEntries) out->rcStop = 1u;
        }
    }
    __syncthreads();
    if (total > maxEntries) return;
    for (uint32_t i = threadIdx.x; i < C; i += blockDim.x) {
        const uint32_t r = (uint32_t)(key[i] >> 14), b = rowPtr[r], len = rowPtr[r + 1] - b;
        for (uint32_t k = 0; k < len; ++k) {
            const long long d = (long long)colInd[b + k] - (long long)r;
            if (d < INT32_MIN || d > INT32_MAX) out->rcStop = 1u;
            delta[off[i] + k] = (int32_t)d;
            tval[off[i] + k] = val[b + k];
        }
    }
}

// cls[row]: the row's slot in, its class id out; mask[row] (optional) the class's mask. *differ is set
// when a row is not the class its hash says.
__global__ void __launch_bounds__(kBlock) k_class_assign(uint32_t nrow,
                                                         const uint32_t* __restrict__ rowPtr,
                                                         const uint32_t* __restrict__ colInd,
                                                         const double* __restrict__ val,
                                                         const uint16_t* __restrict__ idOf,
                                                         const uint32_t* __restrict__ off,
                                                         const int32_t* __restrict__ delta,
                                                         const double* __restrict__ tval,
                                                         const uint16_t* __restrict__ classMask,
                                                         uint16_t* __restrict__ cls,
                                                         uint16_t* __restrict__ mask,
                                                         unsigned* __restrict__ differ)
{
    bool same = true;
    for (size_t row = (size_t)blockIdx.x * blockDim.x + threadIdx.x; row < nrow;
         row += (size_t)gridDim.x * blockDim.x) {
        const uint32_t id = idOf[cls[row]], b = rowPtr[row], len = rowPtr[row + 1] - b;
        const uint32_t t = off[id];
        same = same && off[id + 1] - t == len;
        if (same)
            for (uint32_t k = 0; k < len; ++k)
                same = same && (long long)delta[t + k] == (long long)colInd[b + k] - (long long)row &&
                       __double_as_longlong(tval[t + k]) == __double_as_longlong(val[b + k]);
        cls[row] = (uint16_t)id;
        if (mask) mask[row] = classMask[id];
    }
    if (!same) atomicOr(differ, 1u);
}

// Stencil masks: when the classes' column offsets, taken together, are at most kMaxStencil
// distinct values each carrying one value (bitwise) wherever it occurs, and every class
// lists its offsets in ascending order (the CSR order), each row is a bit mask over that
// sorted offset list. Summing the present entries in list order is the CSR order.
bool class_masks(const std::vector<uint32_t>& off, const std::vector<int32_t>& delta,
                 const std::vector<double>& val, Mat& T, std::vector<uint16_t>& cm)
{
    std::map<int32_t, double> U;
    const uint32_t C = (uint32_t)off.size() - 1;
    for (uint32_t c = 0; c < C; ++c)
        for (uint32_t k = off[c]; k < off[c + 1]; ++k) {
            if (k > off[c] && delta[k] <= delta[k - 1]) return false;
            auto it = U.find(delta[k]);
            if (it == U.end()) {
                if (U.size() == (size_t)kMaxStencil) return false;
                U.emplace(delta[k], val[k]);
            } else if (std::memcmp(&it->second, &val[k], 8) != 0) {
                return false;
            }
        }
    if (U.empty()) return false;
    std::map<int32_t, int> pos;
    T.skLen = 0;
    for (auto& kv : U) {
        pos[kv.first] = (int)T.skLen;
        T.skDelta[T.skLen] = kv.first;
        T.skVal[T.skLen] = kv.second;
        ++T.skLen;
    }
    cm.assign(C, 0);
    for (uint32_t c = 0; c < C; ++c)
        for (uint32_t k = off[c]; k < off[c + 1]; ++k) cm[c] |= (uint16_t)(1u << pos[delta[k]]);
    return true;
}

// Device memory of one upload's temporaries.
struct Slab {
    void* p = nullptr;
    ~Slab() { dev_free(p); }
};

constexpr unsigned long long kClassSeeds[3] = {1469598103934665603ull, 0x9e3779b97f4a7c15ull,
                                               0xd1b54a32d192ed03ull};

} // namespace

void m_free(Mat& M)
{
    dev_free(M.rowPtr);
    dev_free(M.colInd);
    dev_free(M.diagPtr);
    dev_free(M.val);
    dev_free(M.val32);
    dev_free(M.diag);
    dev_free(M.rcCls);
    dev_free(M.rcOff);
    dev_free(M.rcDelta);
    dev_free(M.rcVal);
    dev_free(M.rcVal32);
    dev_free(M.skMask);
    dev_free(M.cd16);
    M = Mat();
}

namespace {

enum Classes { kBuilt, kUnfit, kCollision };

// The class form of T from the slots that k_class_hash wrote (S, T.rcCls). *what: built, not
// representable, or a hash that different rows share.
int finish_classes(Mat& T, const ClassSlots* S, Inspect* ins, cudaStream_t s, Classes* what)
{
    struct Small {
        uint16_t idOf[kRcSlots];
        uint16_t cm[kRcMaxClasses];
        uint32_t off[kRcMaxClasses + 1];
        unsigned differ;
    };
    *what = kUnfit;
    const size_t cap = std::min<size_t>(std::max<size_t>(64, T.nnz / 8),
                                        (size_t)kRcMaxClasses * kRcMaxRowLen);
    const size_t dOff = (sizeof(Small) + 15) & ~(size_t)15,
                 vOff = (dOff + cap * 4 + 15) & ~(size_t)15;
    Slab slab;
    int e;
    if ((e = dmalloc(&slab.p, vOff + cap * 8, s))) return e;
    Small* t = (Small*)slab.p;
    int32_t* delta = (int32_t*)((char*)slab.p + dOff);
    double* tval = (double*)((char*)slab.p + vOff);
    k_class_table<<<1, 1024, 0, s>>>(T.rowPtr, T.colInd, T.val, S, (uint32_t)cap, t->idOf, t->off,
                                     delta, tval, ins);
    FB_CUDA(cudaGetLastError());
    Inspect h;
    FB_CUDA(cudaMemcpyAsync(&h, ins, sizeof(h), cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if (h.rcStop) return kOk;
    const uint32_t C = h.classes, E = h.entries;
    std::vector<uint32_t> off((size_t)C + 1);
    std::vector<int32_t> hd(E);
    std::vector<double> hv(E);
    FB_CUDA(cudaMemcpyAsync(off.data(), t->off, ((size_t)C + 1) * 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaMemcpyAsync(hd.data(), delta, (size_t)E * 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaMemcpyAsync(hv.data(), tval, (size_t)E * 8, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    std::vector<uint16_t> cm;
    const bool masks = class_masks(off, hd, hv, T, cm);
    if ((e = dmalloc((void**)&T.rcOff, ((size_t)C + 1) * 4, s)) ||
        (e = dmalloc((void**)&T.rcDelta, (size_t)E * 4 + 16, s)) ||
        (e = dmalloc((void**)&T.rcVal, (size_t)E * 8 + 16, s)) ||
        (masks && (e = dmalloc((void**)&T.skMask, (size_t)T.nrow * 2 + 16, s))))
        return e;
    FB_CUDA(cudaMemcpyAsync(T.rcOff, t->off, ((size_t)C + 1) * 4, cudaMemcpyDeviceToDevice, s));
    FB_CUDA(cudaMemcpyAsync(T.rcDelta, delta, (size_t)E * 4, cudaMemcpyDeviceToDevice, s));
    FB_CUDA(cudaMemcpyAsync(T.rcVal, tval, (size_t)E * 8, cudaMemcpyDeviceToDevice, s));
    if (masks)
        FB_CUDA(cudaMemcpyAsync(t->cm, cm.data(), (size_t)C * 2, cudaMemcpyHostToDevice, s));
    FB_CUDA(cudaMemsetAsync(&t->differ, 0, 4, s));
    k_class_assign<<<std::max(1, std::min(ceil_div(T.nrow, kBlock), 148 * 8)), kBlock, 0, s>>>(
        T.nrow, T.rowPtr, T.colInd, T.val, t->idOf, T.rcOff, T.rcDelta, T.rcVal, t->cm, T.rcCls,
        T.skMask, &t->differ);
    FB_CUDA(cudaGetLastError());
    unsigned differ = 0;
    FB_CUDA(cudaMemcpyAsync(&differ, &t->differ, 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s)); // the host vectors and the slab are done with
    *what = differ ? kCollision : kBuilt;
    T.rcClasses = C;
    T.rcEntries = E;
    return kOk;
}

void drop_classes(Mat& T)
{
    dev_free(T.rcCls);
    dev_free(T.rcOff);
    dev_free(T.rcDelta);
    dev_free(T.rcVal);
    dev_free(T.skMask);
    T.rcCls = T.skMask = nullptr;
    T.rcOff = nullptr;
    T.rcDelta = nullptr;
    T.rcVal = nullptr;
    T.rcClasses = T.rcEntries = T.skLen = 0;
}

} // namespace

// One pass over the structure and, for short rows, one over the entries, both enqueued before
// the single wait for their outcome. Reading the arrays back to check them, find the diagonal
// and hash the rows on one host thread took 10-30 ms on matrices of 2-6 M entries that these
// passes go through in 30-60 us.
int m_inspect(Mat& T, bool classes, cudaStream_t s)
{
    struct Work {
        ClassSlots slots;
        Inspect    ins;
    };
    const uint32_t nrow = T.nrow, nnz = T.nnz;
    const int grid = std::max(1, std::min(ceil_div(nrow, kBlock), 148 * 8));
    Slab slab;
    int e;
    if ((e = dmalloc(&slab.p, sizeof(Work), s)) || (e = dmalloc((void**)&T.diagPtr, (size_t)nrow * 4, s)) ||
        (e = dmalloc((void**)&T.diag, (size_t)nrow * 8, s)))
        return e;
    Work* w = (Work*)slab.p;
    T.meanRowLen = (double)nnz / nrow;
    T.lanes = lanes_for(T.meanRowLen);
    classes = classes && T.val && T.lanes == 1 && nrow <= 0x7fffffffu;
    Inspect h{};
    h.dmin = ~0ull;
    FB_CUDA(cudaMemcpyAsync(&w->ins, &h, sizeof(h), cudaMemcpyHostToDevice, s));
    k_inspect<<<grid, kBlock, 0, s>>>(nrow, T.mcol, nnz, T.rowPtr, T.colInd, T.val, T.diagPtr,
                                      T.diag, &w->ins);
    FB_CUDA(cudaGetLastError());
    Classes what = kUnfit;
    int attempt = 0;
    do {
        if (classes) {
            if ((e = dmalloc((void**)&T.rcCls, (size_t)nrow * 2 + 16, s))) return e;
            FB_CUDA(cudaMemsetAsync(w->slots.key, 0, sizeof(w->slots.key), s));
            FB_CUDA(cudaMemsetAsync(w->slots.rep, 0xff, sizeof(w->slots.rep), s));
            FB_CUDA(cudaMemsetAsync(&w->ins.classes, 0, 4, s));
            if (nrow > 2 * kRcSample)
                k_class_hash<<<kRcSample / kBlock, kBlock, 0, s>>>(
                    nrow, ceil_div(nrow, kRcSample), nnz, T.rowPtr, T.colInd, T.val,
                    kClassSeeds[attempt], &w->slots, T.rcCls, &w->ins);
            k_class_hash<<<grid, kBlock, 0, s>>>(nrow, 1, nnz, T.rowPtr, T.colInd, T.val,
                                                 kClassSeeds[attempt], &w->slots, T.rcCls, &w->ins);
            FB_CUDA(cudaGetLastError());
        }
        FB_CUDA(cudaMemcpyAsync(&h, &w->ins, sizeof(h), cudaMemcpyDeviceToHost, s));
        FB_CUDA(cudaStreamSynchronize(s));
        if (h.bad) return kErrMatData;
        if (classes && !h.rcStop && (e = finish_classes(T, &w->slots, &w->ins, s, &what))) return e;
        if (what != kBuilt) drop_classes(T);
    } while (what == kCollision && ++attempt < 3); // three shared hashes: the CSR form stays
    T.rcOn = what == kBuilt;
    T.maxRowLen = h.maxLen;
    T.tileSpan = h.span[0];
    std::memcpy(T.laneSpan, h.span, sizeof(T.laneSpan));
    T.near16 = !h.far16;
    T.diagConst = false;
    if (T.val && nrow == T.mcol && !h.noDiag && h.dmin == h.dmax) {
        std::memcpy(&T.diagValue, &h.dmin, 8);
        T.diagConst = T.diagValue != 0.0;
    }
    return kOk;
}

int m_adopt(Mat& M, Mat& T, cudaStream_t s)
{
    cudaGetDevice(&T.dev);
    int e = T.nrow == 0 || T.mcol == 0 || T.nnz == 0 ? kErrMatSize : m_inspect(T, true, s);
    if (!e && cudaStreamSynchronize(s) != cudaSuccess) e = kErrCuda;
    if (e) {
        cudaStreamSynchronize(s);
        m_free(T);
        return e;
    }
    M = T;
    return kOk;
}

int after_legacy_stream(cudaStream_t s)
{
    cudaEvent_t ev;
    FB_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ev, cudaStreamLegacy);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, ev, 0);
    cudaEventDestroy(ev);
    FB_CUDA(e);
    return kOk;
}

int m_upload(Mat& M, uint32_t nrow, uint32_t mcol, uint32_t nnz, const uint32_t* rowPtr,
             const uint32_t* colInd, const double* values, bool hostPtrs, cudaStream_t s)
{
    if (nrow == 0 || mcol == 0 || nnz == 0) return kErrMatSize;
    Mat T;
    T.nrow = nrow;
    T.mcol = mcol;
    T.nnz = nnz;
    cudaGetDevice(&T.dev);
    int e;
    auto fill = [&]() -> int {
        const cudaMemcpyKind kind = hostPtrs ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
        if ((e = dmalloc((void**)&T.rowPtr, ((size_t)nrow + 1) * 4, s)) ||
            (e = dmalloc((void**)&T.colInd, (size_t)nnz * 4, s)) ||
            (values && (e = dmalloc((void**)&T.val, (size_t)nnz * 8, s))))
            return e;
        // device arrays may still be being written by work on the legacy default stream
        // (torch's, say): the copies wait for it, as a blocking copy there would
        if (!hostPtrs && (e = after_legacy_stream(s))) return e;
        FB_CUDA(cudaMemcpyAsync(T.rowPtr, rowPtr, ((size_t)nrow + 1) * 4, kind, s));
        FB_CUDA(cudaMemcpyAsync(T.colInd, colInd, (size_t)nnz * 4, kind, s));
        if (values) FB_CUDA(cudaMemcpyAsync(T.val, values, (size_t)nnz * 8, kind, s));
        if ((e = m_inspect(T, true, s))) return e;
        FB_CUDA(cudaStreamSynchronize(s));
        return kOk;
    };
    if ((e = fill())) {
        cudaStreamSynchronize(s); // nothing of this call still runs on arrays that now go
        m_free(T);
        return e;
    }
    M = T;
    return kOk;
}

// ---- 16-bit column offsets ------------------------------------------------------------------
// cd16[k] = colInd[k] - row(k) when every entry is within 32,767 columns of its row (banded
// FDM/FEM matrices up to bandwidths of 32,767, the 128^3 Laplacian's is 16,384): the
// thread-per-row kernels then read 2 bytes per entry instead of 4 and form the column by one
// add, with the entries and their order unchanged -- the same results bit for bit. Formed
// when they are first turned on: they are off by default, and forming them for every matrix
// cost 49 us and an allocation on a 6M-entry upload.
__global__ void k_col16(uint32_t nrow, const uint32_t* __restrict__ rowPtr,
                        const uint32_t* __restrict__ colInd, int16_t* __restrict__ out)
{
    for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrow;
         r += (size_t)gridDim.x * blockDim.x)
        for (uint32_t k = rowPtr[r]; k < rowPtr[r + 1]; ++k)
            out[k] = (int16_t)((long long)colInd[k] - (long long)r);
}

int m_build_col16(Mat& M, cudaStream_t s)
{
    if (!M.near16 || M.cd16) return kOk;
    int e;
    if ((e = dmalloc((void**)&M.cd16, ((size_t)M.nnz + 8) * 2, s))) return e;
    k_col16<<<std::max(1, std::min(ceil_div(M.nrow, kBlock), 148 * 8)), kBlock, 0, s>>>(
        M.nrow, M.rowPtr, M.colInd, M.cd16);
    FB_CUDA(cudaGetLastError());
    FB_CUDA(cudaStreamSynchronize(s));
    return kOk;
}

} // namespace fb
