// spmv.cu -- CSRx matrices in HBM: SpMV (MAT::Apply), residual (MAT::Residual), the
// lanes-per-row autotuner and the sampled outer product of the adjoint gradient.
//
// SpMV mapping: a group of L lanes (L = 1, 2, ..., 32) owns one row; the lanes stride over
// the row's entries so that a warp reads 32/L consecutive rows' values and column indices
// as one contiguous, coalesced stream; x is gathered through L1/L2 (the stencil rows touch
// nearby columns, so x stays cache resident). L = 1 is the scalar thread-per-row kernel and
// L = 32 the warp-per-row vector kernel; L is chosen from the mean row length or timed.
#include <algorithm>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "internal.h"

namespace fb {

constexpr int kSlotResidualXinf = kSlots - 1;
constexpr int kTileLanes = 4; // lanes a row of k_lane_tiles (mean rows of 17 to 32 entries)

// y = A x (RES: r = b - A x, with the x ~ 0 shortcut of MAT::Residual) on stencil masks of
// the fixed 5- or 7-point shape (SH), W consecutive rows per thread (stencil_group).
template <typename T, int SH, bool RES>
__global__ void __launch_bounds__(kBlock) k_stencil_vec(CSRView<T> A, const T* __restrict__ x,
                                                        const T* __restrict__ b,
                                                        T* __restrict__ y,
                                                        const double* __restrict__ xinf)
{
    using VT = Vec16<T>;
    using V = typename VT::V;
    constexpr int W = VT::W;
    const bool shortcut = RES && *xinf < kCloseZero;
    const uint32_t nw = A.nrow / W, stride = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31u;
    const V* xv = reinterpret_cast<const V*>(x);
    const V* bv = reinterpret_cast<const V*>(b);
    V* yv = reinterpret_cast<V*>(y);
    // the loop bound is the same on every lane of a warp (all lanes shuffle)
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g - lane < nw; g += stride) {
        const bool act = g < nw;
        T s[W];
#pragma unroll
        for (int j = 0; j < W; ++j) s[j] = T(0);
        if (!shortcut) {
            V c;
            stencil_group<T, SH>(A, g, nw, act, [&](uint32_t h) { return xv[h]; }, c, s);
        }
        if (act) {
            if (RES) {
                const V bb = bv[g];
#pragma unroll
                for (int j = 0; j < W; ++j) s[j] = VT::at(bb, j) - s[j];
            }
            yv[g] = VT::make(s);
        }
    }
}


template <typename T, int L, bool PAT>
__global__ void __launch_bounds__(kBlock) k_spmv(CSRView<T> A, const T* __restrict__ x,
                                                 T* __restrict__ y)
{
    if (L == 1) { // thread per row, or warp tiles of plain CSR: short rows (stencils)
        for_rows<T, PAT>(A, [&](uint32_t j) { return x[j]; }, [&](size_t r, T s) { y[r] = s; });
        return;
    }
    const int lane = threadIdx.x & (L - 1);
    const size_t warpRows = 32 / L;
    const size_t gw = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t nwarps = ((size_t)gridDim.x * blockDim.x) >> 5;
    const size_t sub = (threadIdx.x & 31) / L;
    for (size_t base = gw * warpRows; base < A.nrow; base += nwarps * warpRows) {
        const size_t r = base + sub;
        T s = T(0);
        if (r < A.nrow) {
            const uint32_t b = A.rowPtr[r], e = A.rowPtr[r + 1];
            for (uint32_t k = b + lane; k < e; k += L) {
                const T xv = x[ld_stream(A.colInd + k)];
                s = PAT ? s + xv : fma(ld_stream(A.val + k), xv, s);
            }
        }
        s = group_sum<L>(s);
        if (lane == 0 && r < A.nrow) y[r] = s;
    }
}

// r = b - A x, or r = b when the device flag says NormInf(x) < CLOSE_ZERO (MAT.cxx:459-462).
template <typename T, int L>
__global__ void __launch_bounds__(kBlock) k_residual(CSRView<T> A, const T* __restrict__ b,
                                                     const T* __restrict__ x,
                                                     T* __restrict__ r,
                                                     const double* __restrict__ xinf)
{
    const bool shortcut = *xinf < kCloseZero;
    if (L == 1) {
        if (shortcut) {
            for (size_t row = (size_t)blockIdx.x * blockDim.x + threadIdx.x; row < A.nrow;
                 row += (size_t)gridDim.x * blockDim.x)
                r[row] = b[row] - T(0);
        } else {
            for_rows<T, false>(A, [&](uint32_t j) { return x[j]; },
                               [&](size_t row, T s) { r[row] = b[row] - s; });
        }
        return;
    }
    const int lane = threadIdx.x & (L - 1);
    const size_t warpRows = 32 / L;
    const size_t gw = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t nwarps = ((size_t)gridDim.x * blockDim.x) >> 5;
    const size_t sub = (threadIdx.x & 31) / L;
    for (size_t base = gw * warpRows; base < A.nrow; base += nwarps * warpRows) {
        const size_t row = base + sub;
        T s = T(0);
        if (row < A.nrow && !shortcut) {
            const uint32_t bb = A.rowPtr[row], e = A.rowPtr[row + 1];
            for (uint32_t k = bb + lane; k < e; k += L) s = fma(A.val[k], x[A.colInd[k]], s);
        }
        s = group_sum<L>(s);
        if (lane == 0 && row < A.nrow) r[row] = b[row] - s;
    }
}

// y = A x (RES: r = b - A x, or r = b by the shortcut) with kTileLanes threads a row and the entries
// through shared memory in block tiles: the sums of the lane kernels. Kernels of their own: as a
// branch inside k_spmv and k_residual they cost the lane kernels up to 7% where no tile is taken.
template <bool RES>
__global__ void __launch_bounds__(kBlock) k_lane_tiles(CSRView<double> A, const double* __restrict__ b,
                                                       const double* __restrict__ x,
                                                       double* __restrict__ y,
                                                       const double* __restrict__ xinf)
{
    if (RES && *xinf < kCloseZero) {
        for (size_t row = (size_t)blockIdx.x * blockDim.x + threadIdx.x; row < A.nrow;
             row += (size_t)gridDim.x * blockDim.x)
            y[row] = b[row] - 0.0;
        return;
    }
    csr_tile_rows<double, false, kTileLanes>(
        A, *reinterpret_cast<TileSmem<double>*>(fb_tile_smem), [&](uint32_t j) { return x[j]; },
        [&](size_t row, double s) { y[row] = RES ? b[row] - s : s; });
}

static int spmv_grid(const Ctx& c, uint32_t nrow, int L)
{
    long long threads = (long long)nrow * L;
    long long g = (threads + kBlock - 1) / kBlock;
    long long cap = (long long)c.nsm * 8; // resident at 2048 threads per SM
    return (int)std::max<long long>(1, std::min(g, cap));
}

// Lanes per row from the mean row length: one thread per row up to 16 entries (measured
// fastest for 5- and 7-point stencils on B200), then about 8 entries per lane.
int lanes_for(double mean)
{
    if (mean <= 16) return 1;
    int L = 2;
    while (L < 32 && L * 8 < mean) L *= 2;
    return L;
}

// k_lane_tiles takes FP64 matrices of rows of 20 entries and more on four lanes (64 rows of more
// than 28 do not fit a stage) whose entries take more than kLaneTileBytes, so that one product and
// the next (A and its transpose, say) do not find each other's matrix in the 126 MB L2. Measured
// on B200, lanes and tiles, Apply back to back / Apply, Residual and MultTransposeAdd in turn, us:
// 571,000 rows of 23 entries 41.3 / 161 and 38.9 / 131; 238,000 of 23 (65 MB) 22.2 / 84 and 20.1 /
// 69; 230,000 of 20 (55 MB) 28.8 / 103 and 27.6 / 96. Below: 176,000 of 23 (48 MB) 16.9 / 55 and
// 16.5 / 57; 46,700 of 22 6.3 / 27 and 8.1 / 31; 300,000 of 18 in a band 16.5 and 18.6. More lanes:
// 30,000 rows of 100 (16 lanes) 16 and 18.7, of 200 (32 lanes) 25 and 33.
constexpr unsigned long long kLaneTileBytes = 50ull << 20;

template <typename T>
static bool lane_tiles(Ctx& c, CSRView<T>& A, int L, uint32_t span, const void* kern, size_t* smem,
                       int* grid)
{
    if (sizeof(T) != 8 || L != kTileLanes || !A.val || A.nnz < 20ull * A.nrow ||
        A.nnz * 12ull < kLaneTileBytes)
        return false;
    *smem = with_tiles(A, kBlock, span);
    if (*smem && tiles_fit(kern, *smem)) {
        *grid = std::min(ceil_div((long long)A.nrow * kTileLanes, kBlock),
                         resident_grid(c, kern, kBlock, *smem));
        return true;
    }
    A.tiles = 0;
    return false;
}

template <typename T>
static int launch_spmv(Ctx& c, CSRView<T> A, int L, uint32_t span, const T* x, T* y)
{
    if (A.nrow == 0) return kOk;
    const int need = spmv_grid(c, A.nrow, L);
    const bool pat = A.val == nullptr && !A.gnz;
    if (L == 1 && !pat) {
        const int sh = stencil_vec_shape(A, x, y, x);
        if (sh) {
            auto gv = [&](auto kern) {
                const int g = std::min(need, resident_grid(c, (const void*)kern, kBlock));
                kern<<<g, kBlock, 0, c.stream>>>(A, x, (const T*)nullptr, y, (const double*)nullptr);
            };
            ++c.launches;
            if (sh == 5)
                gv(k_stencil_vec<T, 5, false>);
            else
                gv(k_stencil_vec<T, 7, false>);
            FB_CUDA(cudaGetLastError());
            return kOk;
        }
    }
    if constexpr (std::is_same<T, double>::value) {
        size_t smem = 0;
        int g = 0;
        if (lane_tiles(c, A, L, span, (const void*)k_lane_tiles<false>, &smem, &g)) {
            ++c.launches;
            k_lane_tiles<false><<<g, kBlock, smem, c.stream>>>(A, nullptr, x, y, nullptr);
            FB_CUDA(cudaGetLastError());
            return kOk;
        }
    }
    const size_t tiles = L == 1 ? with_tiles(A, kBlock, span) : 0;
    auto go = [&](auto kern) {
        CSRView<T> V = A;
        size_t smem = tiles;
        if (smem && !tiles_fit((const void*)kern, smem)) V.tiles = 0, smem = 0;
        const int g = std::min(need, resident_grid(c, (const void*)kern, kBlock, smem));
        kern<<<g, kBlock, smem, c.stream>>>(V, x, y);
    };
#define SPMV_CASE(LL)                                                                     \
    case LL:                                                                              \
        if (pat)                                                                          \
            go(k_spmv<T, LL, true>);                                                      \
        else                                                                              \
            go(k_spmv<T, LL, false>);                                                     \
        break;
    ++c.launches;
    switch (L) {
        SPMV_CASE(1)
        SPMV_CASE(2)
        SPMV_CASE(4)
        SPMV_CASE(8)
        SPMV_CASE(16)
        SPMV_CASE(32)
        default: return kErrInputPar;
    }
#undef SPMV_CASE
    FB_CUDA(cudaGetLastError());
    return kOk;
}

int m_spmv(Ctx& c, const Mat& A, const double* x, double* y)
{
    return launch_spmv<double>(c, A.v64(), A.lanes, A.span(A.lanes), x, y);
}

int m_spmv32(Ctx& c, const Mat& A, const float* x, float* y)
{
    return launch_spmv<float>(c, A.v32(), A.lanes, A.span(A.lanes), x, y);
}

// *mark = 1.0 when some |x_i| is not below CLOSE_ZERO (NormInf(x) >= CLOSE_ZERO, a NaN counting
// as below as in VEC::NormInf), else 0.0: all that MAT::Residual's shortcut asks. Every block
// looks at the same kBlock entries spread over x; where one of them decides, the first block
// writes the mark and nobody reads or reduces anything else. Only a (nearly) zero or very sparse x
// is read on, by each thread up to its first such entry, eight loads at a time. NormInf itself read
// all of it: 11 of the 100 us of a residual at 160^3, now 5; a blocking residual of x = 0 there 30.2
// us (29.2 with NormInf, 35 with a vote of the block after every load), at 250^3 78 (77, 93).
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mark_above(uint32_t n, const T* __restrict__ x, Scratch s,
                                                       double* mark)
{
    auto above = [](T v) { return (double)fabs(v) >= kCloseZero; };
    if (__syncthreads_or(n && above(x[(size_t)threadIdx.x * n / kBlock]))) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *mark = 1.0;
        return;
    }
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    bool found = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n && !found; i += 8 * stride) {
        T v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = i + u * stride < n ? x[i + u * stride] : T(0);
#pragma unroll
        for (int u = 0; u < 8; ++u) found = found || above(v[u]);
    }
    double acc[1] = {found ? 1.0 : 0.0};
    const int ops[1] = {kMax};
    grid_reduce<1>(acc, ops, s, [=] __device__(const double* t) { *mark = t[0]; });
}

template <typename T>
static int residual_t(Ctx& c, const Mat& A, CSRView<T> V, const T* b, const T* x, T* r,
                      const double* xinf)
{
    if (A.nrow == 0) return kOk;
    if (!V.val && !V.gnz) return kErrMatData; // MAT::Residual reads values (MAT.cxx:466)
    if (!xinf) {
        double* mark = c.dslot + kSlotResidualXinf;
        ++c.launches;
        k_mark_above<T><<<c.grid(A.mcol, kBlock), kBlock, 0, c.stream>>>(A.mcol, x, c.red, mark);
        FB_CUDA(cudaGetLastError());
        xinf = mark;
    }
    const int need = spmv_grid(c, A.nrow, A.lanes);
    if (A.lanes == 1) {
        const int sh = stencil_vec_shape(V, x, b, r);
        if (sh) {
            auto gv = [&](auto kern) {
                const int g = std::min(need, resident_grid(c, (const void*)kern, kBlock));
                kern<<<g, kBlock, 0, c.stream>>>(V, x, b, r, xinf);
            };
            ++c.launches;
            if (sh == 5)
                gv(k_stencil_vec<T, 5, true>);
            else
                gv(k_stencil_vec<T, 7, true>);
            FB_CUDA(cudaGetLastError());
            return kOk;
        }
    }
    if constexpr (std::is_same<T, double>::value) {
        size_t smem = 0;
        int g = 0;
        if (lane_tiles(c, V, A.lanes, A.span(A.lanes), (const void*)k_lane_tiles<true>, &smem, &g)) {
            ++c.launches;
            k_lane_tiles<true><<<g, kBlock, smem, c.stream>>>(V, b, x, r, xinf);
            FB_CUDA(cudaGetLastError());
            return kOk;
        }
    }
    const size_t tiles = A.lanes == 1 ? with_tiles(V, kBlock) : 0;
    auto go = [&](auto kern) {
        CSRView<T> W = V;
        size_t smem = tiles;
        if (smem && !tiles_fit((const void*)kern, smem)) W.tiles = 0, smem = 0;
        const int g = std::min(need, resident_grid(c, (const void*)kern, kBlock, smem));
        kern<<<g, kBlock, smem, c.stream>>>(W, b, x, r, xinf);
    };
    ++c.launches;
    switch (A.lanes) {
        case 1: go(k_residual<T, 1>); break;
        case 2: go(k_residual<T, 2>); break;
        case 4: go(k_residual<T, 4>); break;
        case 8: go(k_residual<T, 8>); break;
        case 16: go(k_residual<T, 16>); break;
        default: go(k_residual<T, 32>); break;
    }
    FB_CUDA(cudaGetLastError());
    return kOk;
}

int m_residual(Ctx& c, const Mat& A, const double* b, const double* x, double* r,
               const double* xinf)
{
    return residual_t<double>(c, A, A.v64(), b, x, r, xinf);
}

int m_residual(Ctx& c, const Mat& A, const float* b, const float* x, float* r,
               const double* xinf)
{
    if (!A.val && !A.grid) return kErrMatData;
    return residual_t<float>(c, A, A.v32(), b, x, r, xinf);
}

// ---- setup-time kernels ----------------------------------------------------------------

__global__ void k_to_f32(size_t n, const double* __restrict__ a, float* __restrict__ b)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

unsigned tile_timeouts_spmv() { return tile_timeouts(); }

int Mat::ensure32(cudaStream_t s)
{
    if (!val) return kOk;
    int e;
    if (!val32) {
        if ((e = dmalloc((void**)&val32, (size_t)nnz * 4, s))) return e;
        k_to_f32<<<std::max(1, std::min(ceil_div(nnz, kBlock), 148 * 8)), kBlock, 0, s>>>(
            nnz, val, val32);
        FB_CUDA(cudaGetLastError());
    }
    if (rcVal && !rcVal32) {
        if ((e = dmalloc((void**)&rcVal32, (size_t)rcEntries * 4 + 16, s))) return e;
        k_to_f32<<<std::max(1, std::min(ceil_div(rcEntries, kBlock), 148 * 8)), kBlock, 0, s>>>(
            rcEntries, rcVal, rcVal32);
        FB_CUDA(cudaGetLastError());
    }
    return kOk;
}

// ---- autotuner: time each lanes-per-row choice on this matrix ---------------------------
int m_autotune(Ctx& c, Mat& A)
{
    if (A.grid) return kOk; // grid operators run thread per row (lanes = 1) only
    double *x = nullptr, *y = nullptr;
    int e;
    if ((e = dmalloc((void**)&x, (size_t)A.mcol * 8, c.stream)) || (e = dmalloc((void**)&y, (size_t)A.nrow * 8, c.stream))) {
        dev_free(x);
        return e;
    }
    FB_CUDA(cudaMemsetAsync(x, 0, (size_t)A.mcol * 8, c.stream));
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    float best = 1e30f;
    int bestL = A.lanes;
    const int orig = A.lanes;
    for (int L = 1; L <= 32; L *= 2) {
        if (L > 2 * (int)A.maxRowLen && L > 1) break;
        A.lanes = L;
        for (int w = 0; w < 2; ++w) m_spmv(c, A, x, y);
        cudaEventRecord(t0, c.stream);
        for (int r = 0; r < 5; ++r) m_spmv(c, A, x, y);
        cudaEventRecord(t1, c.stream);
        cudaEventSynchronize(t1);
        float ms = 0;
        cudaEventElapsedTime(&ms, t0, t1);
        if (ms < best) {
            best = ms;
            bestL = L;
        }
    }
    A.lanes = cudaGetLastError() == cudaSuccess ? bestL : orig;
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    dev_free(x);
    dev_free(y);
    return kOk;
}

// ---- sampled outer product: dA_k = scale * lam[row(k)] * x[col(k)] ----------------------
__global__ void k_sampled_outer(CSRView<double> A, const double* __restrict__ lam,
                                const double* __restrict__ x, double scale,
                                double* __restrict__ dA)
{
    // one warp per 32 rows' worth of entries: lanes stride the contiguous entry range
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.nrow;
         i += (size_t)gridDim.x * blockDim.x) {
        const double li = scale * lam[i];
        for (uint32_t k = A.rowPtr[i]; k < A.rowPtr[i + 1]; ++k) dA[k] = li * x[A.colInd[k]];
    }
}

int m_sampled_outer(Ctx& c, const Mat& A, const double* lam, const double* x, double scale,
                    double* dA)
{
    if (A.grid) return kErrInputPar; // no stored entries to differentiate
    const int g = std::max(1, std::min(ceil_div(A.nrow, kBlock), c.nsm * 8));
    k_sampled_outer<<<g, kBlock, 0, c.stream>>>(A.v64(), lam, x, scale, dA);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

// ---- MAT::MultTransposeAdd: v = A^T v1 + v2 (MAT.cxx:541-606) ---------------------------
// T is A's exact transpose (m_transpose, the order of MAT::TransInPlace). As the reference,
// each v[i] starts from v2[i] and adds the products of row i of T left to right, each
// product rounded before the add (no fused multiply-add), so the results are the
// reference's bit for bit wherever its loop bounds are right (structurally symmetric A).
// Pattern-only matrices count every stored entry as 1, as MAT::Apply does; a grid operator
// walks its stencil points in ascending offset, which is its CSR order.
// Rows of some 20 to 50 entries stream through block tiles of 256 / L rows (csr_tile_rows with
// separately rounded sums) in a kernel of their own: thread per row straight from global memory
// reads words 12 len bytes apart. On B200, thread per row and tiles, us back to back: 571,000 rows
// of 23 entries 64.0 and 48.8, 300,000 of 32 in a band 82.5 and 61.4, 50,000 of 48 39 and 20.7,
// 46,700 of 22 10.4 and 8.5; with scattered columns 600,000 of 30 133 and 121, 150,000 of 30 34.8
// and 36.7. Shorter rows keep the plain loop: 300,000 of 18 18.6 and 21.2, 200,000 of 10 8.3 and
// 10.4, seven entries (160^3) 73 and 76; so do rows whose tiles do not fit a stage on 8 lanes. As
// a branch in the plain kernel the tiles cost it up to 19% there (5,000 rows of 1,000: 161 and 191).
template <bool PAT, int L>
__global__ void __launch_bounds__(kBlock) k_mult_transpose_add_tiles(CSRView<double> T,
                                                                     const double* __restrict__ v1,
                                                                     const double* __restrict__ v2,
                                                                     double* __restrict__ v)
{
    auto from = [&](size_t i) { return v2[i]; };
    csr_tile_rows<double, PAT, L>(T, *reinterpret_cast<TileSmem<double>*>(fb_tile_smem),
                                  [&](uint32_t j) { return v1[j]; },
                                  [&](size_t i, double s) { v[i] = s; },
                                  RowSep<decltype(from)>{from});
}

template <bool GRID, bool PAT>
__global__ void k_mult_transpose_add(CSRView<double> T, const double* __restrict__ v1,
                                     const double* __restrict__ v2, double* __restrict__ v)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < T.nrow;
         i += (size_t)gridDim.x * blockDim.x) {
        double acc = v2[i];
        if (GRID) {
            const uint32_t m = grid_mask(T, (uint32_t)i);
            for (uint32_t k = 0; k < T.ulen; ++k)
                if ((m >> k) & 1u)
                    acc = __dadd_rn(acc, __dmul_rn(v1[(long long)i + T.udelta[k]], T.uval[k]));
        } else {
            const uint32_t b = T.rowPtr[i], e = T.rowPtr[i + 1];
            for (uint32_t k = b; k < e; ++k)
                acc = __dadd_rn(acc, PAT ? v1[T.colInd[k]]
                                         : __dmul_rn(v1[T.colInd[k]], T.val[k]));
        }
        v[i] = acc;
    }
}

int m_mult_transpose_add(Ctx& c, const Mat& T, const double* v1, const double* v2, double* v)
{
    if (T.nrow == 0) return kOk;
    CSRView<double> V = T.view<double>(T.val, nullptr);
    V.cd16 = nullptr;
    auto plain = [&](auto kern) {
        const int g = std::max(1, std::min(ceil_div(T.nrow, kBlock), c.nsm * 8));
        kern<<<g, kBlock, 0, c.stream>>>(V, v1, v2, v);
    };
    // the fewest threads a row whose tiles fit a stage
    int L = 1;
    while (L < 8 && T.span(L) > TileShape<double>::cap) L *= 2;
    const size_t smem = T.grid || L == 1 || T.nnz < 20ull * T.nrow
                            ? 0
                            : with_tiles(V, kBlock, T.span(L));
    auto tiled = [&](auto kern) {
        const int g = std::min(ceil_div((long long)T.nrow * L, kBlock),
                               resident_grid(c, (const void*)kern, kBlock, smem));
        if (!tiles_fit((const void*)kern, smem)) return false;
        kern<<<g, kBlock, smem, c.stream>>>(V, v1, v2, v);
        return true;
    };
    auto by = [&](auto PAT) {
        constexpr bool P = decltype(PAT)::value;
        if (smem && (L == 2   ? tiled(k_mult_transpose_add_tiles<P, 2>)
                     : L == 4 ? tiled(k_mult_transpose_add_tiles<P, 4>)
                              : tiled(k_mult_transpose_add_tiles<P, 8>)))
            return;
        V.tiles = 0;
        plain(k_mult_transpose_add<false, P>);
    };
    if (T.grid)
        plain(k_mult_transpose_add<true, false>);
    else if (!T.val)
        by(std::true_type{});
    else
        by(std::false_type{});
    FB_CUDA(cudaGetLastError());
    return kOk;
}

// ---- structured-grid (matrix-free) operators --------------------------------------------
// The GPU counterpart of the reference's matrix-free LOP example (example/TestMatFree.cxx:
// 26-176): y = A x on an nx x ny x nz grid with a constant-coefficient stencil, Dirichlet
// truncation at the faces, without any stored matrix. Rows are grid points in x-fastest
// order; a row's entries are the stencil points inside the grid in ascending column order,
// so every kernel computes exactly what it computes on the assembled CSR matrix.

__global__ void k_fill_const(uint32_t n, double v, double* __restrict__ y)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        y[i] = v;
}

int m_create_stencil(Mat& M, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t npts,
                     const int32_t* dx, const int32_t* dy, const int32_t* dz, const double* coef,
                     cudaStream_t s)
{
    if (!dx || !dy || !dz || !coef) return kErrInputPar;
    if (nx == 0 || ny == 0 || nz == 0) return kErrMatSize;
    const uint64_t n64 = (uint64_t)nx * ny * nz;
    if (n64 > 0xffffffffull || (uint64_t)nx * ny > 0xffffffffull) return kErrMatSize;
    if (npts == 0 || npts > (uint32_t)kMaxStencil) return kErrInputPar;
    struct Pt {
        int64_t flat;
        int32_t d[3];
        double  v;
    };
    std::vector<Pt> pts(npts);
    for (uint32_t k = 0; k < npts; ++k) {
        const int32_t d[3] = {dx[k], dy[k], dz[k]};
        for (int a = 0; a < 3; ++a)
            if (d[a] < -3 || d[a] > 3) return kErrInputPar; // reach of at most 3 points
        pts[k] = Pt{(int64_t)d[0] + (int64_t)nx * ((int64_t)d[1] + (int64_t)ny * d[2]),
                    {d[0], d[1], d[2]}, coef[k]};
    }
    // points that reach past the grid in some dimension are never inside it: dropped (in a
    // grid one point thick, such points could share a flattened offset with real ones)
    const uint32_t ext[3] = {nx, ny, nz};
    pts.erase(std::remove_if(pts.begin(), pts.end(),
                             [&](const Pt& p) {
                                 for (int a = 0; a < 3; ++a)
                                     if ((uint32_t)std::abs(p.d[a]) >= ext[a]) return true;
                                 return false;
                             }),
              pts.end());
    npts = (uint32_t)pts.size();
    // a present neighbour (ix + dx, iy + dy, iz + dz) is column row + flat, so ascending
    // flattened offset is the CSR column order of every row
    std::sort(pts.begin(), pts.end(), [](const Pt& a, const Pt& b) { return a.flat < b.flat; });
    for (uint32_t k = 1; k < npts; ++k)
        if (pts[k].flat == pts[k - 1].flat) return kErrInputPar;
    Mat T;
    T.grid = true;
    T.nrow = T.mcol = (uint32_t)n64;
    T.gdim[0] = nx;
    T.gdim[1] = ny;
    T.gdim[2] = nz;
    T.skLen = npts;
    uint64_t nnz = 0;
    double diagv = 0.0;
    bool hasDiag = false;
    for (uint32_t k = 0; k < npts; ++k) {
        T.skDelta[k] = (int32_t)pts[k].flat;
        T.skVal[k] = pts[k].v;
        uint64_t cnt = 1;
        for (int a = 0; a < 3; ++a) {
            T.gd[a][k] = (int8_t)pts[k].d[a];
            const uint32_t r = (uint32_t)std::abs(pts[k].d[a]);
            cnt *= r < ext[a] ? ext[a] - r : 0;
        }
        nnz += cnt;
        if (pts[k].flat == 0) {
            hasDiag = true;
            diagv = pts[k].v;
        }
    }
    if (nnz > 0xffffffffull) return kErrMatSize;
    T.nnz = (uint32_t)nnz;
    T.lanes = 1;
    T.maxRowLen = npts;
    T.meanRowLen = (double)nnz / (double)n64;
    T.diagConst = hasDiag && diagv != 0.0;
    T.diagValue = diagv;
    cudaGetDevice(&T.dev);
    int e;
    if ((e = dmalloc((void**)&T.diag, (size_t)T.nrow * 8, s))) return e;
    k_fill_const<<<std::max(1, std::min(ceil_div(T.nrow, kBlock), 148 * 8)), kBlock, 0, s>>>(
        T.nrow, diagv, T.diag);
    FB_CUDA(cudaGetLastError());
    FB_CUDA(cudaStreamSynchronize(s));
    M = T;
    return kOk;
}

void m_grid_csr(const Mat& M, std::vector<uint32_t>& rowPtr, std::vector<uint32_t>& colInd,
                std::vector<double>& values)
{
    const uint32_t nx = M.gdim[0], ny = M.gdim[1], nz = M.gdim[2];
    rowPtr.assign((size_t)M.nrow + 1, 0);
    colInd.clear();
    values.clear();
    colInd.reserve(M.nnz);
    values.reserve(M.nnz);
    uint32_t row = 0;
    for (uint32_t iz = 0; iz < nz; ++iz)
        for (uint32_t iy = 0; iy < ny; ++iy)
            for (uint32_t ix = 0; ix < nx; ++ix, ++row) {
                for (uint32_t k = 0; k < M.skLen; ++k) {
                    const int64_t jx = (int64_t)ix + M.gd[0][k], jy = (int64_t)iy + M.gd[1][k],
                                  jz = (int64_t)iz + M.gd[2][k];
                    if (jx < 0 || jy < 0 || jz < 0 || jx >= nx || jy >= ny || jz >= nz) continue;
                    colInd.push_back((uint32_t)((int64_t)row + M.skDelta[k]));
                    values.push_back(M.skVal[k]);
                }
                rowPtr[(size_t)row + 1] = (uint32_t)colInd.size();
            }
}

} // namespace fb
