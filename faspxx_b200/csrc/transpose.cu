// transpose.cu -- CSR -> CSC in exactly MAT::TransInPlace's order (src/MAT.cxx:479-538): the
// entries of a column in the order of their CSR positions, which is ascending rows.
//
// Column counts by atomics, which also give every entry a slot in its column, a scan, a
// scatter of whole entries as 16-byte records into those slots, and the records of each column
// put in order of position (k_rank_rows; columns longer than kRankMost: keys sorted, values
// gathered by position).
#include "segsort.cuh"

namespace fb {
namespace {

__global__ void k_col_count(uint32_t nnz, const uint32_t* __restrict__ colInd,
                            uint32_t* __restrict__ cnt, uint32_t* __restrict__ slot)
{
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
         k += (size_t)gridDim.x * blockDim.x)
        slot[k] = atomicAdd(&cnt[colInd[k]], 1u);
}

__global__ void __launch_bounds__(256) k_longest(uint32_t n, const uint32_t* __restrict__ cnt,
                                                 unsigned* __restrict__ longest)
{
    unsigned m = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        m = max(m, cnt[i]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(longest, m);
}

// Entry k of row i, column c -> record (row, position, value), or key, at tRowPtr[c] + slot[k].
// A block takes 256 rows, whose entries are contiguous, and its threads stride over the
// entries, finding an entry's row by a search of the block's row pointers.
template <bool REC>
__global__ void __launch_bounds__(kBlock) k_scatter_cols(
    uint32_t nrow, const uint32_t* __restrict__ rowPtr, const uint32_t* __restrict__ colInd,
    const double* __restrict__ val, const uint32_t* __restrict__ tRowPtr,
    const uint32_t* __restrict__ slot, Rec* __restrict__ rec, uint64_t* __restrict__ keys)
{
    __shared__ uint32_t rp[kBlock + 1];
    const size_t nt = ((size_t)nrow + kBlock - 1) / kBlock;
    for (size_t tile = blockIdx.x; tile < nt; tile += gridDim.x) {
        const uint32_t r0 = (uint32_t)(tile * kBlock);
        const uint32_t rows = nrow - r0 < (uint32_t)kBlock ? nrow - r0 : (uint32_t)kBlock;
        __syncthreads();
        for (uint32_t t = threadIdx.x; t <= rows; t += kBlock) rp[t] = rowPtr[(size_t)r0 + t];
        __syncthreads();
        for (size_t k = (size_t)rp[0] + threadIdx.x; k < rp[rows]; k += kBlock) {
            uint32_t lo = 0, hi = rows;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (rp[mid] <= k)
                    lo = mid;
                else
                    hi = mid;
            }
            const size_t o = (size_t)tRowPtr[colInd[k]] + slot[k];
            if (REC) {
                Rec r;
                r.col = r0 + lo;
                r.pos = (uint32_t)k;
                r.val = val ? val[k] : 0.0;
                rec[o] = r;
            } else {
                keys[o] = (uint64_t)(r0 + lo) << 32 | (uint32_t)k;
            }
        }
    }
}

__global__ void k_take(uint32_t nnz, const uint64_t* __restrict__ keys, const double* __restrict__ val,
                       uint32_t* __restrict__ tColInd, double* __restrict__ tVal)
{
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < nnz;
         q += (size_t)gridDim.x * blockDim.x) {
        tColInd[q] = (uint32_t)(keys[q] >> 32);
        if (tVal) tVal[q] = val[(uint32_t)keys[q]];
    }
}

// The transpose of a grid operator is the grid operator with every offset negated (the
// same coefficients), in ascending order of the negated flattened offsets.
static int grid_transpose(Ctx& c, const Mat& A, Mat& T)
{
    std::vector<int32_t> dx(A.skLen), dy(A.skLen), dz(A.skLen);
    for (uint32_t k = 0; k < A.skLen; ++k) {
        dx[k] = -A.gd[0][k];
        dy[k] = -A.gd[1][k];
        dz[k] = -A.gd[2][k];
    }
    return m_create_stencil(T, A.gdim[0], A.gdim[1], A.gdim[2], A.skLen, dx.data(), dy.data(),
                            dz.data(), A.skVal, c.stream);
}

// R's sizes, rowPtr, colInd and val.
int transpose_arrays(Ctx& c, const Mat& A, Mat& R)
{
    const uint32_t m = A.mcol, n = A.nrow, nnz = A.nnz;
    cudaStream_t s = c.stream;
    Tmp t(s);
    R.nrow = m;
    R.mcol = n;
    R.nnz = nnz;
    R.dev = A.dev;
    uint32_t *cnt = nullptr, *slot = nullptr, *tiles = nullptr;
    unsigned* longest = nullptr;
    int e;
    if ((e = dmalloc((void**)&R.rowPtr, ((size_t)m + 1) * 4, s)) ||
        (e = dmalloc((void**)&R.colInd, (size_t)nnz * 4, s)) ||
        (A.val && (e = dmalloc((void**)&R.val, (size_t)nnz * 8, s))) || (e = t.get(&cnt, m)) ||
        (e = t.get(&slot, nnz)) || (e = t.get(&tiles, (m + (size_t)kTile - 1) / kTile)) ||
        (e = t.get(&longest, 1)))
        return e;
    FB_CUDA(cudaMemsetAsync(cnt, 0, (size_t)m * 4, s));
    FB_CUDA(cudaMemsetAsync(longest, 0, 4, s));
    k_col_count<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, A.colInd, cnt, slot);
    k_longest<<<grid_for(m, 256), 256, 0, s>>>(m, cnt, longest);
    FB_CUDA(cudaGetLastError());
    if ((e = scan_counts(s, m, cnt, R.rowPtr, tiles))) return e;
    unsigned most = 0;
    FB_CUDA(cudaMemcpyAsync(&most, longest, 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    const int g = std::max(1, std::min(ceil_div(n, kBlock), c.nsm * 8));
    Rec* rec = nullptr;
    if (most <= kRankMost && !t.get(&rec, nnz)) { // without memory for records: keys, half as long
        k_scatter_cols<true><<<g, kBlock, 0, s>>>(n, A.rowPtr, A.colInd, A.val, R.rowPtr, slot, rec,
                                                  nullptr);
        FB_CUDA(cudaGetLastError());
        return rank_rows<false>(c, m, R.rowPtr, nullptr, R.rowPtr, nullptr, RecSource{rec}, R.colInd,
                                R.val);
    }
    uint64_t* keys = nullptr;
    if ((e = t.get(&keys, nnz))) return e;
    k_scatter_cols<false><<<g, kBlock, 0, s>>>(n, A.rowPtr, A.colInd, A.val, R.rowPtr, slot, nullptr,
                                               keys);
    FB_CUDA(cudaGetLastError());
    if ((e = sort_row_keys(c, t, m, R.rowPtr, keys, nnz))) return e;
    k_take<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, keys, A.val, R.colInd, R.val);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

} // namespace

int m_transpose(Ctx& c, const Mat& A, Mat& T)
{
    if (A.grid) return grid_transpose(c, A, T);
    Mat R;
    int e = transpose_arrays(c, A, R);
    if (!e) e = m_inspect(R, false, c.stream);
    if (e) {
        cudaStreamSynchronize(c.stream);
        m_free(R);
        return e;
    }
    R.diagConst = false; // the solvers on a transpose read its diagonal vector
    R.diagValue = 0.0;
    R.lanes = A.lanes;
    T = R;
    return kOk;
}

} // namespace fb
