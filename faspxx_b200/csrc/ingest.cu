// ingest.cu -- a CSRx matrix built on the device from the arrays that FASP++'s file readers
// produce, with the conversions of ReadMat (src/ReadData.cxx:361-446) done as GPU scans and
// sorts instead of host loops:
//
//   MatrixMarket triplets, 0-based (ReadMTX, ReadData.cxx:98-218), then MTXtoMAT
//   (src/MATUtil.cxx:416-436): MTXtoCSR's counting sort by row (:252-300), SortCSRRow
//   (:439-476), CSRtoMAT (:303-413);
//
//   raw CSR arrays (ReadCSR, ReadData.cxx:221-358): the 1-based shift (:350-353), then
//   SortCSRRow and CSRtoMAT as ReadMat's .csr branch does (ReadData.cxx:376-400).
//
// The order both reference paths produce, and this file reproduces: rows ascending; in a
// row, columns ascending, and entries with equal columns (duplicates are kept, not summed)
// in input order, since the counting sort and the insertion sort are both stable. A row
// without a diagonal entry gets an explicit 0.0 at its sorted place.
//
// Entries are ordered by (column, input position), which is unique, so any correct order of
// a row's entries is the stable one. Rows of up to kRankMost entries: each triplet goes into
// its row as a 16-byte record (the slot comes from the counting pass) and one kernel puts a
// row's records in order, diagonals inserted (k_rank_rows). A matrix with a longer row carries
// every entry as one 64-bit key (column << 32 | input position) and gathers the value
// through the position at the end; keys are sorted by length class: groups of 8 or 32 lanes with a
// register bitonic network (short rows), one block with a shared-memory bitonic network per
// segment of up to 4096 keys, and merge passes (rank by binary search) above that.
#include <algorithm>
#include <vector>

#include "segsort.cuh"

namespace fb {
namespace {

// What the counting pass tells the host.
struct Counted {
    int                bad;    // an index out of range, or rows that are not CSR
    unsigned           maxLen; // longest row, its diagonal included
    unsigned long long added;  // diagonals to insert
};

// ---- input checks (CheckCSR, MATUtil.cxx:110-174, before any indexed access) and row lengths --

// cnt[r] entries of row r, each triplet's slot in its row (the order inside a row is
// arbitrary here and fixed later by (column, position)), and the rows with a diagonal entry.
__global__ void k_count_coo(uint32_t nnz, uint32_t nrow, uint32_t mcol,
                            const uint32_t* __restrict__ rowInd, const uint32_t* __restrict__ colInd,
                            uint32_t* __restrict__ cnt, uint32_t* __restrict__ slot,
                            uint8_t* __restrict__ has, Counted* __restrict__ out)
{
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz;
         j += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = rowInd[j], c = colInd[j];
        if (r >= nrow || c >= mcol) {
            out->bad = 1;
            continue;
        }
        slot[j] = atomicAdd(&cnt[r], 1u);
        if (r == c) has[r] = 1;
    }
}

// Row pointers start at 0, or at 1 for 1-based files (ReadCSR shifts those,
// ReadData.cxx:350-353); monotone; rowPtr[nrow] - rowPtr[0] == nnz; shifted columns < mcol. Rows of
// up to kCountLong entries a thread each, longer ones the whole block (a row of 8,000,000 on one
// thread took 170 ms).
constexpr uint32_t kCountLong = 128;

__global__ void __launch_bounds__(kBlock) k_count_csr(uint32_t nrow, uint32_t mcol, uint32_t nnz,
                            const uint32_t* __restrict__ rowPtr, const uint32_t* __restrict__ colInd,
                            uint32_t* __restrict__ cnt, uint8_t* __restrict__ has,
                            Counted* __restrict__ out)
{
    __shared__ uint32_t lrow[kBlock], nlong;
    const uint32_t base = rowPtr[0];
    bool bad = base > 1u || rowPtr[nrow] - base != nnz || rowPtr[nrow] < base;
    for (size_t i0 = (size_t)blockIdx.x * kBlock; i0 < nrow && base <= 1u;
         i0 += (size_t)gridDim.x * kBlock) {
        const size_t i = i0 + threadIdx.x;
        if (threadIdx.x == 0) nlong = 0;
        __syncthreads();
        uint32_t b = 0, e = 0;
        if (i < nrow) {
            b = rowPtr[i] - base;
            e = rowPtr[i + 1] - base;
            if (b > e || e > nnz) { // not CSR: its entries are not looked at
                bad = true;
                e = b;
            }
            cnt[i] = e - b;
        }
        if (e - b > kCountLong) {
            lrow[atomicAdd(&nlong, 1u)] = (uint32_t)i;
        } else if (i < nrow) {
            bool diag = false;
            for (uint32_t k = b; k < e; ++k) {
                const uint32_t c = colInd[k] - base; // a 0 in a 1-based file wraps and fails too
                bad = bad || c >= mcol;
                diag = diag || c == i;
            }
            has[i] = diag ? 1 : 0;
        }
        __syncthreads();
        for (uint32_t l = 0; l < nlong; ++l) {
            const uint32_t r = lrow[l], rb = rowPtr[r] - base, re = rowPtr[(size_t)r + 1] - base;
#pragma unroll 4
            for (size_t k = (size_t)rb + threadIdx.x; k < re; k += kBlock) {
                const uint32_t c = colInd[k] - base;
                bad = bad || c >= mcol;
                if (c == r) has[r] = 1; // 0 before
            }
        }
        __syncthreads();
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) out->bad = 1;
}

// len[i] = row i's entries with its diagonal, miss[i] = whether that is to be inserted (in: has[i]);
// a row >= mcol without one fails (CheckCSR rejects the inserted column).
__global__ void __launch_bounds__(256) k_row_len(uint32_t nrow, uint32_t mcol,
                                                 const uint32_t* __restrict__ cnt,
                                                 uint8_t* __restrict__ miss,
                                                 uint32_t* __restrict__ len,
                                                 Counted* __restrict__ out)
{
    unsigned maxLen = 0, added = 0;
    bool bad = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nrow;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t m = miss[i] ? 0u : 1u;
        miss[i] = (uint8_t)m;
        len[i] = cnt[i] + m;
        maxLen = max(maxLen, len[i]);
        added += m;
        bad = bad || (m && i >= mcol);
    }
    maxLen = __reduce_max_sync(0xffffffffu, maxLen);
    added = __reduce_add_sync(0xffffffffu, added);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out->maxLen, maxLen);
        if (added) atomicAdd(&out->added, (unsigned long long)added);
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) out->bad = 1;
}

// ---- entries in row segments ----------------------------------------------------------------

// MTXtoCSR step 3 (MATUtil.cxx:278-286): the whole entry moves, so nothing is gathered by
// position later (a random 8-byte read per entry).
__global__ void k_scatter_rec(uint32_t nnz, const uint32_t* __restrict__ rowInd,
                              const uint32_t* __restrict__ colInd, const double* __restrict__ values,
                              const uint32_t* __restrict__ rowPtr, const uint32_t* __restrict__ slot,
                              Rec* __restrict__ rec)
{
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz;
         j += (size_t)gridDim.x * blockDim.x) {
        Rec r;
        r.col = colInd[j];
        r.pos = (uint32_t)j;
        r.val = values[j];
        rec[(size_t)rowPtr[rowInd[j]] + slot[j]] = r;
    }
}

__global__ void k_scatter_keys(uint32_t nnz, const uint32_t* __restrict__ rowInd,
                               const uint32_t* __restrict__ colInd, const uint32_t* __restrict__ rowPtr,
                               const uint32_t* __restrict__ slot, uint64_t* __restrict__ keys)
{
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz;
         j += (size_t)gridDim.x * blockDim.x)
        keys[(size_t)rowPtr[rowInd[j]] + slot[j]] = (uint64_t)colInd[j] << 32 | (uint64_t)j;
}

__global__ void k_keys_csr(uint32_t nrow, uint32_t nnz, const uint32_t* __restrict__ rowPtr,
                           const uint32_t* __restrict__ colInd, uint32_t* __restrict__ rowPtr0,
                           uint64_t* __restrict__ keys)
{
    const uint32_t base = rowPtr[0];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i <= nrow;
         i += (size_t)gridDim.x * blockDim.x)
        rowPtr0[i] = rowPtr[i] - base;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
         k += (size_t)gridDim.x * blockDim.x)
        keys[k] = (uint64_t)(colInd[k] - base) << 32 | (uint64_t)k;
}

// ---- CSRtoMAT: explicit zero diagonals (MATUtil.cxx:303-413) ----------------------------------

// Keys of row i with column below i, in a sorted row.
__device__ __forceinline__ uint32_t below_diag(const uint64_t* keys, uint32_t b, uint32_t e, uint32_t i)
{
    return count_below(keys + b, e - b, (uint64_t)i << 32);
}

__global__ void k_gather(uint32_t nrow, uint32_t nnz, const uint32_t* __restrict__ rowPtr,
                         const uint32_t* __restrict__ rowPtr2, const uint8_t* __restrict__ miss,
                         const uint64_t* __restrict__ keys, const double* __restrict__ values,
                         uint32_t* __restrict__ colInd2, double* __restrict__ val2)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t p = tid; p < nnz; p += stride) {
        uint32_t lo = 0, hi = nrow; // the row r with rowPtr[r] <= p < rowPtr[r + 1]
        while (hi - lo > 1) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (rowPtr[mid] <= p)
                lo = mid;
            else
                hi = mid;
        }
        const uint64_t k = keys[p];
        const uint32_t col = (uint32_t)(k >> 32);
        const size_t q =
            (size_t)rowPtr2[lo] + (p - rowPtr[lo]) + (miss[lo] && col > lo ? 1u : 0u);
        colInd2[q] = col;
        val2[q] = values[(uint32_t)k];
    }
    for (size_t i = tid; i < nrow; i += stride)
        if (miss[i]) {
            const uint32_t b = rowPtr[i], e = rowPtr[i + 1];
            const size_t q = (size_t)rowPtr2[i] + below_diag(keys, b, e, (uint32_t)i);
            colInd2[q] = (uint32_t)i;
            val2[q] = 0.0;
        }
}

// The row lengths of cnt with the diagonals that miss (in: the rows that have one) lacks, their
// scan into T.rowPtr and the matrix's arrays. *maxLen: the longest row.
int lay_out(Ctx& c, Tmp& t, uint32_t nrow, uint32_t mcol, uint32_t nnz, const uint32_t* cnt,
            uint8_t* miss, Counted* out, uint32_t* tiles, Mat& T, uint32_t* maxLen)
{
    cudaStream_t s = c.stream;
    int e;
    uint32_t* len = nullptr;
    if ((e = t.get(&len, nrow)) || (e = dmalloc((void**)&T.rowPtr, ((size_t)nrow + 1) * 4, s)))
        return e;
    k_row_len<<<grid_for(nrow, 256), 256, 0, s>>>(nrow, mcol, cnt, miss, len, out);
    FB_CUDA(cudaGetLastError());
    if ((e = scan_counts(s, nrow, len, T.rowPtr, tiles))) return e;
    Counted h;
    FB_CUDA(cudaMemcpyAsync(&h, out, sizeof(h), cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if (h.bad) return kErrMatData;
    const uint64_t nnz2 = (uint64_t)nnz + h.added;
    if (nnz2 > 0xffffffffull) return kErrMatSize;
    T.nrow = nrow;
    T.mcol = mcol;
    T.nnz = (uint32_t)nnz2;
    *maxLen = h.maxLen;
    if ((e = dmalloc((void**)&T.colInd, (size_t)nnz2 * 4, s))) return e;
    return dmalloc((void**)&T.val, (size_t)nnz2 * 8, s);
}

// A matrix with long rows: sorts the rows of keys (row segments given by the 0-based rowPtr,
// on the device), inserts the missing diagonals and gathers the values.
int sorted_rows(Ctx& c, Tmp& t, uint32_t nrow, uint32_t nnz, const uint32_t* rowPtr,
                uint64_t* keys, const double* values, const uint8_t* miss, Mat& T)
{
    int e;
    if ((e = sort_row_keys(c, t, nrow, rowPtr, keys, nnz))) return e;
    k_gather<<<grid_for(std::max<size_t>(nnz, nrow), 256), 256, 0, c.stream>>>(
        nrow, nnz, rowPtr, T.rowPtr, miss, keys, values, T.colInd, T.val);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

int coo_arrays(Ctx& c, uint32_t nrow, uint32_t mcol, uint32_t nnz, const uint32_t* rowInd,
               const uint32_t* colInd, const double* values, bool onDevice, Mat& T)
{
    cudaStream_t s = c.stream;
    Tmp t(s);
    int e;
    const uint32_t *ri = nullptr, *ci = nullptr;
    const double* va = nullptr;
    if ((onDevice && (e = after_legacy_stream(s))) ||
        (e = stage(t, s, rowInd, nnz, onDevice, &ri)) || (e = stage(t, s, colInd, nnz, onDevice, &ci)) ||
        (e = stage(t, s, values, nnz, onDevice, &va)))
        return e;
    Counted* out = nullptr;
    uint32_t *cnt = nullptr, *slot = nullptr, *tiles = nullptr, maxLen = 0;
    uint8_t* miss = nullptr;
    if ((e = t.get(&out, 1)) || (e = t.get(&cnt, nrow)) || (e = t.get(&miss, nrow)) ||
        (e = t.get(&slot, nnz)) || (e = t.get(&tiles, (nrow + (size_t)kTile - 1) / kTile)))
        return e;
    FB_CUDA(cudaMemsetAsync(out, 0, sizeof(Counted), s));
    FB_CUDA(cudaMemsetAsync(cnt, 0, (size_t)nrow * 4, s));
    FB_CUDA(cudaMemsetAsync(miss, 0, nrow, s));
    k_count_coo<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, nrow, mcol, ri, ci, cnt, slot, miss, out);
    FB_CUDA(cudaGetLastError());
    if ((e = lay_out(c, t, nrow, mcol, nnz, cnt, miss, out, tiles, T, &maxLen))) return e;
    Rec* rec = nullptr;
    if (maxLen <= kRankMost && !t.get(&rec, T.nnz)) { // without memory for records: keys, half as long
        k_scatter_rec<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, ri, ci, va, T.rowPtr, slot, rec);
        FB_CUDA(cudaGetLastError());
        return rank_rows<true>(c, nrow, T.rowPtr, nullptr, T.rowPtr, miss, RecSource{rec}, T.colInd,
                               T.val);
    }
    uint32_t* rp = nullptr;
    uint64_t* keys = nullptr;
    if ((e = t.get(&rp, (size_t)nrow + 1)) || (e = t.get(&keys, nnz)) ||
        (e = scan_counts(s, nrow, cnt, rp, tiles)))
        return e;
    k_scatter_keys<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, ri, ci, rp, slot, keys);
    FB_CUDA(cudaGetLastError());
    return sorted_rows(c, t, nrow, nnz, rp, keys, va, miss, T);
}

int csr_arrays(Ctx& c, uint32_t nrow, uint32_t mcol, uint32_t nnz, const uint32_t* rowPtr,
               const uint32_t* colInd, const double* values, bool onDevice, Mat& T)
{
    cudaStream_t s = c.stream;
    Tmp t(s);
    int e;
    const uint32_t *rpIn = nullptr, *ci = nullptr;
    const double* va = nullptr;
    if ((onDevice && (e = after_legacy_stream(s))) ||
        (e = stage(t, s, rowPtr, (size_t)nrow + 1, onDevice, &rpIn)) ||
        (e = stage(t, s, colInd, nnz, onDevice, &ci)) || (e = stage(t, s, values, nnz, onDevice, &va)))
        return e;
    Counted* out = nullptr;
    uint32_t *cnt = nullptr, *tiles = nullptr, maxLen = 0;
    uint8_t* miss = nullptr;
    if ((e = t.get(&out, 1)) || (e = t.get(&cnt, nrow)) || (e = t.get(&miss, nrow)) ||
        (e = t.get(&tiles, (nrow + (size_t)kTile - 1) / kTile)))
        return e;
    FB_CUDA(cudaMemsetAsync(out, 0, sizeof(Counted), s));
    FB_CUDA(cudaMemsetAsync(miss, 0, nrow, s));
    k_count_csr<<<grid_for(nrow, 256), 256, 0, s>>>(nrow, mcol, nnz, rpIn, ci, cnt, miss, out);
    FB_CUDA(cudaGetLastError());
    if ((e = lay_out(c, t, nrow, mcol, nnz, cnt, miss, out, tiles, T, &maxLen))) return e;
    if (maxLen <= kRankMost)
        return rank_rows<false>(c, nrow, rpIn, rpIn, T.rowPtr, miss, CsrSource{ci, va, rpIn},
                                T.colInd, T.val);
    uint32_t* rp = nullptr;
    uint64_t* keys = nullptr;
    if ((e = t.get(&rp, (size_t)nrow + 1)) || (e = t.get(&keys, nnz))) return e;
    k_keys_csr<<<grid_for(std::max(nnz, nrow + 1u), 256), 256, 0, s>>>(nrow, nnz, rpIn, ci, rp, keys);
    FB_CUDA(cudaGetLastError());
    return sorted_rows(c, t, nrow, nnz, rp, keys, va, miss, T);
}

// The arrays that `make` forms, as a matrix.
template <typename F>
int matrix_of(Ctx& c, Mat& M, F&& make)
{
    Mat T;
    const int e = make(T);
    if (e) {
        cudaStreamSynchronize(c.stream);
        m_free(T);
        return e;
    }
    return m_adopt(M, T, c.stream);
}

} // namespace

int m_from_coo(Ctx& c, uint32_t nrow, uint32_t mcol, uint32_t nnz, const uint32_t* rowInd,
               const uint32_t* colInd, const double* values, bool onDevice, Mat& M)
{
    if (!rowInd || !colInd || !values) return kErrInputPar;
    if (nrow == 0 || mcol == 0 || nnz == 0) return kErrMatSize;
    return matrix_of(c, M, [&](Mat& T) {
        return coo_arrays(c, nrow, mcol, nnz, rowInd, colInd, values, onDevice, T);
    });
}

int m_from_csr_raw(Ctx& c, uint32_t nrow, uint32_t mcol, uint32_t nnz, const uint32_t* rowPtr,
                   const uint32_t* colInd, const double* values, bool onDevice, Mat& M)
{
    if (!rowPtr || !colInd || !values) return kErrInputPar;
    if (nrow == 0 || mcol == 0 || nnz == 0) return kErrMatSize;
    return matrix_of(c, M, [&](Mat& T) {
        return csr_arrays(c, nrow, mcol, nnz, rowPtr, colInd, values, onDevice, T);
    });
}

} // namespace fb
