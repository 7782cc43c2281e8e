// mg.cu -- the MG cycle with transfer operators as few launches per level as its data flow allows,
// and Jacobi::Solve on small matrices in shared memory.
//
// A cycle whose smoothers and coarse solver run a fixed number of sweeps (minIter = maxIter) reads
// no norm on the host. As separate kernels a level with two sweeps before and after took some 20
// launches: NormInf(x) for MAT::Residual's shortcut, a residual and an update per sweep (the
// Galerkin levels' rows are longer than one thread takes), vector resets, a product and an
// addition per transfer. Coarse levels are nothing but launch and reduction latency: on B200 a
// V(2,2) cycle took 330 us at 31^3 and 800 us at 127^3. Here a level takes one launch for
// its first two sweeps (from x = 0), one a sweep after that, one residual, one restriction and
// one prolongation that also corrects x; levels of up to 1,024 rows take one launch for all their
// sweeps. Whether NormInf(x) is below CLOSE_ZERO, which a residual's shortcut tests, is a mark that
// the kernel writing x leaves when any |x| is not: the same decision without a reduction.
#include "solver.h"

namespace fb {
namespace {

// Marks *out (0.0 before the cycle) when any thread of the block saw an |x| that is not below
// CLOSE_ZERO: all that a residual's shortcut asks of NormInf(x) (a NaN counts as below, as in
// VEC::NormInf). Every thread calls it.
__device__ __forceinline__ void mark_above(bool above, double* out)
{
    if (__syncthreads_or(above) && threadIdx.x == 0) *out = 1.0;
}

__device__ __forceinline__ bool above_zero(double x) { return fabs(x) >= kCloseZero; }

__device__ __forceinline__ TileSmem<double>& tile_smem()
{
    return *reinterpret_cast<TileSmem<double>*>(fb_tile_smem);
}

// First in a kernel, before it waits for its predecessor: no kernel of a cycle writes a matrix, so
// the block's first tiles are copied while the predecessor still runs. rows_of() takes them, a
// kernel without rows_of() calls no_rows().
template <int L>
__device__ __forceinline__ void tiles_first(const CSRView<double>& A)
{
    if (A.tiles && threadIdx.x == 0) CsrTiles<double, false, L>(A, tile_smem()).begin();
}

template <int L>
__device__ __forceinline__ void no_rows(const CSRView<double>& A)
{
    if (A.tiles && threadIdx.x == 0) CsrTiles<double, false, L>(A, tile_smem()).drain();
}

// Rows of A on L lanes each, in block tiles where the view has them (see tiles_first; both ways
// the same sums): own(row, sum) on the row's first lane. A sweep of the 27-point level of 63^3
// rows took 27.5 us row by row, 22.6 in tiles (cold).
template <int L, typename XV, typename OWN>
__device__ __forceinline__ void rows_of(const CSRView<double>& A, XV xv, OWN own)
{
    if (A.tiles) {
        csr_tile_rows<double, false, L, true>(A, tile_smem(), xv, own);
        return;
    }
    if (L == 1) {
        for_rows<double, false>(A, xv, own);
        return;
    }
    const uint32_t lane = threadIdx.x & (L - 1);
    const size_t stride = (size_t)gridDim.x * blockDim.x / L;
    const size_t first = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / L;
    for (size_t r0 = first - (threadIdx.x & 31) / L; r0 < A.nrow; r0 += stride) { // warp-uniform
        const size_t row = r0 + (threadIdx.x & 31) / L;
        double s = 0.0;
        if (row < A.nrow) {
            const uint32_t b = A.rowPtr[row], e = A.rowPtr[row + 1];
            for (uint32_t k = b + lane; k < e; k += L)
                s = fma(ld_stream(A.val + k), xv(ld_stream(A.colInd + k)), s);
        }
        s = group_sum<L>(s);
        if (lane == 0 && row < A.nrow) own(row, s);
    }
}

// Jacobi's weight / diag: one number where the diagonal is one value (the same bits), else the
// vector. Reading it had been a quarter of a sweep's bytes on a constant stencil.
struct DiagInv {
    const double* v;
    double c;
    __device__ __forceinline__ double operator[](size_t i) const { return v ? v[i] : c; }
};

DiagInv diag_inv(const Pcd& p)
{
    if (p.A->diagConst) return {nullptr, (1.0 / p.A->diagValue) * p.weight};
    return {p.dinv, 0.0};
}

// One Jacobi sweep, xout = xin + dinv .* r with r = b - A xin, or r = b when NormInf(xin) (*in)
// is below CLOSE_ZERO (MAT.cxx:455-476, Iter.cxx:83-92). TWO: the first two sweeps from
// x = 0, whose first is dinv .* b, formed where it is gathered; *in is its mark.
template <int L, bool TWO>
__global__ void __launch_bounds__(kBlock, 5) k_mg_sweep(CSRView<double> A, const double* __restrict__ b,
                                                     const double* __restrict__ xin,
                                                     DiagInv dinv,
                                                     double* __restrict__ xout,
                                                     const double* __restrict__ in, double* out)
{
    tiles_first<L>(A);
    pdl_wait();
    pdl_release();
    const bool shortcut = *in < kCloseZero;
    bool above = false;
    auto x0 = [&](size_t j) { return TWO ? b[j] * dinv[j] : xin[j]; };
    auto own = [&](size_t i, double sum) {
        const double xi = x0(i) + (b[i] - sum) * dinv[i];
        xout[i] = xi;
        above = above || above_zero(xi);
    };
    if (shortcut) {
        no_rows<L>(A);
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.nrow;
             i += (size_t)gridDim.x * blockDim.x)
            own(i, 0.0);
    } else {
        rows_of<L>(A, [&](uint32_t j) { return x0(j); }, own);
    }
    mark_above(above, out);
}

// r = b - A x, or r = b by the same shortcut (MAT.cxx:455-476).
template <int L>
__global__ void __launch_bounds__(kBlock) k_mg_residual(CSRView<double> A,
                                                        const double* __restrict__ b,
                                                        const double* __restrict__ x,
                                                        double* __restrict__ r,
                                                        const double* __restrict__ in)
{
    tiles_first<L>(A);
    pdl_wait();
    pdl_release();
    auto own = [&](size_t i, double s) { r[i] = b[i] - s; };
    if (*in < kCloseZero) {
        no_rows<L>(A);
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.nrow;
             i += (size_t)gridDim.x * blockDim.x)
            own(i, 0.0);
    } else {
        rows_of<L>(A, [&](uint32_t j) { return x[j]; }, own);
    }
}

// The first sweep from x = 0: x = dinv .* b.
__global__ void __launch_bounds__(kBlock) k_mg_first(uint32_t n, const double* __restrict__ b,
                                                     DiagInv dinv,
                                                     double* __restrict__ x, double* out)
{
    pdl_wait();
    pdl_release();
    bool above = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const double xi = b[i] * dinv[i];
        x[i] = xi;
        above = above || above_zero(xi);
    }
    mark_above(above, out);
}

// bc = R r, and the mark of dinv .* bc, the coarse level's first sweep.
template <int L>
__global__ void __launch_bounds__(kBlock) k_mg_restrict(CSRView<double> R, const double* __restrict__ r,
                                                        double* __restrict__ bc,
                                                        DiagInv dinv, double* out)
{
    tiles_first<L>(R);
    pdl_wait();
    pdl_release();
    bool above = false;
    rows_of<L>(R, [&](uint32_t j) { return r[j]; }, [&](size_t i, double s) {
        bc[i] = s;
        above = above || above_zero(s * dinv[i]);
    });
    mark_above(above, out);
}

// x += P e.
template <int L>
__global__ void __launch_bounds__(kBlock) k_mg_correct(CSRView<double> P, const double* __restrict__ e,
                                                       double* __restrict__ x, double* out)
{
    tiles_first<L>(P);
    pdl_wait();
    pdl_release();
    bool above = false;
    rows_of<L>(P, [&](uint32_t j) { return e[j]; }, [&](size_t i, double s) {
        const double xi = x[i] + s;
        x[i] = xi;
        above = above || above_zero(xi);
    });
    mark_above(above, out);
}

// A whole Jacobi::Solve (Iter.cxx:56-112) on at most 1,024 rows, thread per row, with the
// matrix and x in shared memory: a sweep of a 27-row coarsest level waits for shared memory and
// one or two block barriers instead of global loads (40 sweeps: 105 -> 12 us on B200). Rows are
// summed left to right as row_apply sums them. zero: x is taken as 0 and not read. RE: the first
// RE entries of a row stay in registers over the sweeps, whose only loads are then the gathers,
// all in flight at once: 40 sweeps of 27 rows 27 us instead of 35 (cold, with the launch). One warp
// only: with the four warps of 125 rows 40 sweeps took 5 us more than from shared memory.
constexpr int kSmallRegs = 32;

template <typename T, int RE>
__global__ void __launch_bounds__(RE ? kSmallRegs : 1024) k_jacobi_small(uint32_t n, uint32_t nnz,
                                                       const uint32_t* __restrict__ rowPtr,
                                                       const uint32_t* __restrict__ colInd,
                                                       const T* __restrict__ val,
                                                       const T* __restrict__ b, T* __restrict__ x,
                                                       const T* __restrict__ dinv,
                                                       fasp_gpu_params prm, int zero, double* out)
{
    extern __shared__ __align__(16) unsigned char small[];
    __shared__ double sh[32];
    T* sv = reinterpret_cast<T*>(small);
    T* sx = sv + nnz;
    uint16_t* sc = reinterpret_cast<uint16_t*>(sx + n);
    const uint32_t t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
#pragma unroll 8
    for (uint32_t k = t; k < nnz; k += blockDim.x) { // the matrix: no predecessor writes it
        sv[k] = __ldg(val + k);
        sc[k] = (uint16_t)__ldg(colInd + k);
    }
    const bool row = t < n;
    const uint32_t r0 = row ? rowPtr[t] : 0u, r1 = row ? rowPtr[t + 1] : 0u;
    const T di = row ? dinv[t] : T(0);
    pdl_wait();
    pdl_release();
    const T bi = row ? b[t] : T(0);
    T xi = row && !zero ? x[t] : T(0);
    if (row) sx[t] = xi;
    T rv[RE ? RE : 1];
    uint32_t rc[RE ? RE : 1];
    const uint32_t re = min(r1 - r0, (uint32_t)RE);
    if (RE) {
        __syncthreads(); // the entries are in shared memory
#pragma unroll
        for (int u = 0; u < RE; ++u) {
            rv[u] = (uint32_t)u < re ? sv[r0 + u] : T(0);
            rc[u] = (uint32_t)u < re ? sc[r0 + u] : 0u;
        }
    }
    // the block's sum of v, the same on every thread
    auto all = [&](double v) {
        v = warp_reduce(v, kSum);
        __syncthreads();
        if (lane == 0) sh[wid] = v;
        __syncthreads();
        return __shfl_sync(0xffffffffu, warp_reduce(lane < nw ? sh[lane] : 0.0, kSum), 0);
    };
    double denAbs = 1.0;
    bool above = __syncthreads_or(above_zero((double)xi)); // orders the writes of sx too
    for (uint32_t it = 0; it < prm.maxIter; ++it) {
        T s = T(0);
        if (RE && above) {
            T g[RE ? RE : 1];
#pragma unroll
            for (int u = 0; u < RE; ++u) g[u] = sx[rc[u]];
#pragma unroll
            for (int u = 0; u < RE; ++u)
                if ((uint32_t)u < re) s = fma(rv[u], g[u], s);
        }
        if (above)
            for (uint32_t k = r0 + re; k < r1; k += 8) { // eight entries' loads, then their FMAs
                uint32_t c[8];
                T v[8], g[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const bool in = k + u < r1;
                    c[u] = in ? sc[k + u] : 0u;
                    v[u] = in ? sv[k + u] : T(0);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) g[u] = sx[c[u]];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (k + u < r1) s = fma(v[u], g[u], s);
            }
        const T r = bi - s;
        if (it >= prm.minIter) {
            const double resAbs = sqrt(all((double)(row ? r * r : T(0))));
            if (it == prm.minIter) denAbs = (kCloseZero > resAbs) ? kCloseZero : resAbs;
            if (resAbs / denAbs < prm.relTol || resAbs < prm.absTol) break;
        }
        __syncthreads(); // every row's sum has read the old x
        if (row) {
            xi = xi + r * di;
            sx[t] = xi;
        }
        above = __syncthreads_or(above_zero((double)xi));
    }
    if (row) x[t] = xi;
    if (out && t == 0 && above) *out = 1.0;
}

constexpr size_t kSmallBytes = 200 * 1024; // shared memory of k_jacobi_small at most

size_t small_bytes(const Mat& A, size_t elem)
{
    return (size_t)A.nnz * (elem + 2) + (size_t)A.nrow * elem;
}

template <typename F>
void by_lanes(int lanes, F&& go)
{
    switch (lanes) {
        case 1: go(std::integral_constant<int, 1>()); break;
        case 2: go(std::integral_constant<int, 2>()); break;
        case 4: go(std::integral_constant<int, 4>()); break;
        case 8: go(std::integral_constant<int, 8>()); break;
        case 16: go(std::integral_constant<int, 16>()); break;
        default: go(std::integral_constant<int, 32>()); break;
    }
}

// kern(view of A, args...) on one resident wave, rows on `lanes` lanes, in block tiles where A
// takes them.
template <typename... P, typename... X>
int launch_rows(Ctx& c, const Mat& A, int lanes, void (*kern)(CSRView<double>, P...), X... args)
{
    CSRView<double> V = A.v64();
    size_t smem = with_tiles(V, kBlock, A.span(lanes));
    if (smem && !tiles_fit((const void*)kern, smem)) V.tiles = 0, smem = 0;
    const int g = std::min(c.grid((long long)A.nrow * lanes, kBlock),
                           resident_grid(c, (const void*)kern, kBlock, smem));
    ++c.launches;
    FB_CUDA(launch_pdl(kern, dim3((unsigned)g), dim3(kBlock), smem, c.stream, V, args...));
    return kOk;
}

// Lanes for a transfer operator's rows: a matrix without stored values for it (a grid operator)
// keeps one thread per row.
int transfer_lanes(const Mat& A) { return A.grid ? 1 : lanes_for(A.meanRowLen); }

} // namespace

bool jacobi_small_fits(const Mat& A, size_t elem)
{
    return !A.grid && A.val && A.nrow == A.mcol && A.nrow <= 1024 && small_bytes(A, elem) <= kSmallBytes;
}

template <typename T>
int jacobi_small(Ctx& c, const Mat& A, const T* val, const T* b, T* x, const T* dinv,
                 const fasp_gpu_params& prm, bool zero, double* mark)
{
    const size_t smem = small_bytes(A, sizeof(T));
    const auto kern = A.nrow <= kSmallRegs ? k_jacobi_small<T, 32> : k_jacobi_small<T, 0>;
    FB_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmallBytes));
    ++c.launches;
    FB_CUDA(launch_pdl(kern, dim3(1), dim3((A.nrow + 31u) & ~31u), smem, c.stream, A.nrow, A.nnz,
                       (const uint32_t*)A.rowPtr, (const uint32_t*)A.colInd, val, b, x, dinv, prm,
                       zero ? 1 : 0, mark));
    return kOk;
}
template int jacobi_small<double>(Ctx&, const Mat&, const double*, const double*, double*,
                                  const double*, const fasp_gpu_params&, bool, double*);
template int jacobi_small<float>(Ctx&, const Mat&, const float*, const float*, float*, const float*,
                                 const fasp_gpu_params&, bool, double*);

// Marks that one cycle writes: one per kernel that writes x, and one per restriction.
static double cycle_slots(const SolverImpl& S)
{
    double total = 0.0, visits = 1.0;
    for (size_t l = 0; l < S.mgP.size(); ++l) {
        total += visits * (2.0 * S.mgSmooth[l].prm.maxIter + 4.0);
        if (l + 1 < S.mgP.size()) visits *= std::max(1u, S.cfg.mgCycles);
        else total += visits * (S.mgCoarse[l].prm.maxIter + 2.0);
    }
    return total;
}

bool SolverImpl::mg_fixed_cycle() const
{
    if (mgP.empty() || cfg.mgCycles == 0) return false;
    auto fixed = [](const Pcd& p) {
        return p.type == 1 && p.prm.minIter == p.prm.maxIter && p.prm.maxIter >= 1 &&
               (p.A->val || p.A->grid);
    };
    for (size_t l = 0; l < mgP.size(); ++l)
        if (!fixed(mgSmooth[l]) || (l + 1 == mgP.size() && !fixed(mgCoarse[l])) ||
            !(mgP[l]->val || mgP[l]->grid) || !(mgR[l]->val || mgR[l]->grid))
            return false;
    return cycle_slots(*this) <= kMgSlots;
}

// prm.maxIter sweeps of p on b and x. in: the mark of x, or with zero (x is taken as 0 and not
// read) that of dinv .* b where it is known, else null. *end: the mark of the new x.
static int smooth(SolverImpl& S, Pcd& p, const double* b, double* x, bool zero, const double* in,
                  double** end)
{
    Ctx& c = S.c;
    const Mat& A = *p.A;
    const int lanes = A.grid ? 1 : A.lanes;
    int e;
    if (jacobi_small_fits(A, 8)) {
        *end = S.mgInf + S.mgInfUsed++;
        return jacobi_small<double>(c, A, A.val, b, x, p.dinv, p.prm, zero, *end);
    }
    uint32_t left = p.prm.maxIter;
    double *cur = x, *nxt = p.work;
    auto next_slot = [&]() { return *end = S.mgInf + S.mgInfUsed++; };
    if (zero) {
        const bool two = in && left >= 2;
        left -= two ? 2 : 1;
        if (left % 2) std::swap(cur, nxt); // so that the last sweep writes x
        if (two) {
            double* out = next_slot();
            by_lanes(lanes, [&](auto L) {
                e = launch_rows(c, A, lanes, k_mg_sweep<decltype(L)::value, true>, b,
                                (const double*)nullptr, diag_inv(p), cur, in, out);
            });
            if (e) return e;
        } else {
            double* out = next_slot();
            ++c.launches;
            const int g = std::min(c.grid(A.nrow, kBlock),
                                   resident_grid(c, (const void*)k_mg_first, kBlock));
            FB_CUDA(launch_pdl(k_mg_first, dim3((unsigned)g), dim3(kBlock), 0, c.stream, A.nrow, b,
                               diag_inv(p), cur, out));
        }
        in = *end;
    }
    for (; left > 0; --left) {
        double* out = next_slot();
        by_lanes(lanes, [&](auto L) {
            e = launch_rows(c, A, lanes, k_mg_sweep<decltype(L)::value, false>, b, (const double*)cur,
                            diag_inv(p), nxt, in, out);
        });
        if (e) return e;
        in = out;
        std::swap(cur, nxt);
    }
    return cur == x ? (int)kOk : v_copy(c, A.nrow, (const double*)cur, x);
}

// One cycle from level l (MG.cxx:105-152 with this level's operators): pre-smoothing,
// residual, restriction, the coarse solver or the next level's cycles, correction,
// post-smoothing. zero, in, end as in smooth().
static int cycle(SolverImpl& S, uint32_t l, const double* b, double* x, bool zero, const double* in,
                 double** end)
{
    Ctx& c = S.c;
    const uint32_t NL = (uint32_t)S.mgP.size();
    const Mat &A = *S.mgA[l], &R = *S.mgR[l], &P = *S.mgP[l];
    double* r = l == 0 ? S.w[0] : S.mgRes[l];
    int e;
    double* s = nullptr;
    if ((e = smooth(S, S.mgSmooth[l], b, x, zero, in, &s))) return e;
    CSRView<double> V = A.v64();
    if (with_tiles(V, kBlock, A.span(A.lanes)))
        by_lanes(A.lanes, [&](auto L) {
            e = launch_rows(c, A, A.lanes, k_mg_residual<decltype(L)::value>, b, (const double*)x, r,
                            (const double*)s);
        });
    else // stencils keep their row groups
        e = m_residual(c, A, b, (const double*)x, r, (const double*)s);
    if (e) return e;
    Pcd& next = l + 1 == NL ? S.mgCoarse[l] : S.mgSmooth[l + 1];
    double* first = S.mgInf + S.mgInfUsed++;
    const int rl = transfer_lanes(R), pl = transfer_lanes(P);
    by_lanes(rl, [&](auto L) {
        e = launch_rows(c, R, rl, k_mg_restrict<decltype(L)::value>, (const double*)r, S.mgB[l],
                        diag_inv(next), first);
    });
    if (e) return e;
    double* coarse = nullptr;
    if (l + 1 == NL) {
        if ((e = smooth(S, next, S.mgB[l], S.mgX[l], true, first, &coarse))) return e;
    } else {
        for (uint32_t i = 0; i < S.cfg.mgCycles; ++i)
            if ((e = cycle(S, l + 1, S.mgB[l], S.mgX[l], i == 0, i == 0 ? first : coarse, &coarse)))
                return e;
    }
    s = S.mgInf + S.mgInfUsed++;
    by_lanes(pl, [&](auto L) {
        e = launch_rows(c, P, pl, k_mg_correct<decltype(L)::value>, (const double*)S.mgX[l], x, s);
    });
    if (e) return e;
    return smooth(S, S.mgSmooth[l], b, x, false, s, end);
}

int SolverImpl::mg_cycle_fixed(const double* b, double* x, bool zero)
{
    int e;
    if (!mgInf && (e = dev_alloc(&mgInf, sizeof(double) * kMgSlots, c.stream))) return e;
    FB_CUDA(cudaMemsetAsync(mgInf, 0, sizeof(double) * kMgSlots, c.stream));
    mgInfUsed = 0;
    const double* in = nullptr;
    if (!zero) {
        double* xinf = mgInf + mgInfUsed++; // NormInf itself
        if ((e = v_norminf(c, n, (const double*)x, xinf))) return e;
        in = xinf;
    }
    double* end = nullptr;
    return cycle(*this, 0, b, x, zero, in, &end);
}

unsigned tile_timeouts_mg() { return tile_timeouts(); }

} // namespace fb
