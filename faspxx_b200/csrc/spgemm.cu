// spgemm.cu -- sparse matrix algebra on the device: the product C = L R, MAT::Mult
// (src/MAT.cxx:715-800) with its exact result:
//   * the columns of row i of C appear in the order in which the loop over L's row i
//     (entries k in CSR order) and, for each, R's row colInd[k] (entries l in CSR order)
//     first meets them -- MAT::Mult does not sort its rows;
//   * C(i, c) = 0 + sum of L(i,k) R(k,l) over the (k, l) pairs with column c, added in that
//     same loop order, each product rounded before it is added.
// Every (k, l) pair of a row is a candidate. Rows of up to kHashMost candidates: one warp
// per row goes through them 32 at a time in loop order with a hash table of the row's columns
// in shared memory (k_mult_hash). A product with longer rows sorts: the 64-bit keys
// column << 32 | position (position = its index in the loop order) of each row are
// sorted (equal columns become adjacent, in loop order), each run of one column is summed in
// order and remembered by its first position, and a second sort by first position restores
// MAT::Mult's column order. Products are computed and stored before they are added, so no
// multiply-add is fused. Further down: the sum C = a A + b B, MAT::Add.
#include "segsort.cuh"

namespace fb {
namespace {

// The table sizes of k_mult_hash: rows of up to 64, 512 and 2,048 candidates.
constexpr uint32_t kHashCap0 = 64, kHashCap1 = 512, kHashMost = 2048;

// One warp's hash table and the row it forms.
template <uint32_t CAP>
struct HashRow {
    double   acc[CAP];
    uint32_t key[2 * CAP];
    uint32_t col[CAP];
    uint16_t idx[2 * CAP]; // output place of the column at the same hash place
    uint16_t slot[CAP];    // hash place of the column at the same output place
};

struct MultPlan {
    unsigned long long total;   // candidates of the product (can be more than 2^32)
    unsigned           has[4];  // rows in each size class; has[3]: longer ones
};

// candidates per row, their total and the size classes that occur
__global__ void __launch_bounds__(256) k_mult_count(uint32_t n, const uint32_t* __restrict__ lrp,
                                                    const uint32_t* __restrict__ lci,
                                                    const uint32_t* __restrict__ rrp,
                                                    uint32_t* __restrict__ cnt,
                                                    MultPlan* __restrict__ plan)
{
    __shared__ unsigned long long sum;
    unsigned long long mine = 0;
    unsigned has = 0;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        unsigned long long c = 0;
        for (uint32_t k = lrp[i]; k < lrp[i + 1]; ++k) {
            const uint32_t j = lci[k];
            c += rrp[j + 1] - rrp[j];
        }
        cnt[i] = c > 0xffffffffull ? 0xffffffffu : (uint32_t)c;
        mine += c;
        has |= 1u << (c <= kHashCap0 ? 0 : (c <= kHashCap1 ? 1 : (c <= kHashMost ? 2 : 3)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    has = __reduce_or_sync(0xffffffffu, has);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sum, mine);
        for (int k = 0; k < 4; ++k)
            if ((has >> k) & 1u) plan->has[k] = 1u;
    }
    __syncthreads();
    if (threadIdx.x == 0 && sum) atomicAdd(&plan->total, sum);
}

// One warp per row of more than lo and at most CAP candidates. The lanes take 32 candidates
// at a time in loop order (the lane finds its L entry by searching the scan of the R rows'
// lengths). Lanes with the same column are grouped by __match_any_sync; the first of each
// group looks its column up in the row's hash table, and new columns get the next output
// places in lane order, which is the order in which the loop first meets them. Products are
// then added one round per multiplicity, lane order within a column: the loop's order, so
// sums and column order are MAT::Mult's. The row's columns and sums go to its candidates'
// place (coff) in ocol / osum, their number to nout; k_mult_pack closes the gaps.
// Bound by the latency of the dependent loads (row pointer, columns, R's row pointers, R's
// entries): many warps per SM hide it, so the table is no larger than its size class needs.
// Measured on B200, the whole call: R (A P) at 63^3 -> 31^3 (343 candidates a row) 1,530 us
// with the two sorts and their row lists on the host, 285 us this way; A P (24 candidates a
// row) 1,940 and 470 us.
template <uint32_t CAP, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_mult_hash(
    uint32_t n, uint32_t lo, const uint32_t* __restrict__ lrp, const uint32_t* __restrict__ lci,
    const double* __restrict__ lva, const uint32_t* __restrict__ rrp,
    const uint32_t* __restrict__ rci, const double* __restrict__ rva,
    const uint32_t* __restrict__ coff, uint32_t* __restrict__ ocol, double* __restrict__ osum,
    uint32_t* __restrict__ nout)
{
    constexpr uint32_t H = 2 * CAP, kFree = 0xffffffffu; // a column is below mcol <= 2^32 - 1
    extern __shared__ __align__(16) unsigned char hashRows[];
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    HashRow<CAP>& T = reinterpret_cast<HashRow<CAP>*>(hashRows)[threadIdx.x >> 5];
    for (uint32_t h = lane; h < H; h += 32) T.key[h] = kFree;
    __syncwarp();
    const size_t warps = (size_t)gridDim.x * WARPS;
    for (size_t i = (size_t)blockIdx.x * WARPS + (threadIdx.x >> 5); i < n; i += warps) {
        const uint32_t base = coff[i], cand = coff[i + 1] - base;
        if (cand > CAP || (lo && cand <= lo)) continue;
        uint32_t cnt = 0;
        const uint32_t kb = lrp[i], ke = lrp[i + 1];
        for (uint32_t k0 = kb; k0 < ke; k0 += 32) {
            double a = 0.0;
            uint32_t rb = 0, len = 0;
            if (k0 + lane < ke) {
                const uint32_t j = lci[k0 + lane];
                a = lva[k0 + lane];
                rb = rrp[j];
                len = rrp[j + 1] - rb;
            }
            uint32_t S = len; // candidates up to and including this lane's L entry
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, S, o);
                if (lane >= (uint32_t)o) S += y;
            }
            const uint32_t tot = __shfl_sync(0xffffffffu, S, 31);
            const uint32_t first = rb - (S - len); // R entry of candidate p: first + p
            for (uint32_t p0 = 0; p0 < tot; p0 += 32) {
                const uint32_t p = p0 + lane;
                const bool act = p < tot;
                uint32_t own = 0; // the lane whose L entry candidate p belongs to
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const uint32_t v = __shfl_sync(0xffffffffu, S, (int)(own + o - 1));
                    if (v <= p) own += o;
                }
                own = act ? own : lane;
                const double ao = __shfl_sync(0xffffffffu, a, (int)own);
                const uint32_t l = __shfl_sync(0xffffffffu, first, (int)own) + p;
                uint32_t col = 0, peers = 0;
                double prod = 0.0;
                if (act) {
                    col = rci[l];
                    prod = __dmul_rn(ao, rva[l]);
                }
                const uint32_t am = __ballot_sync(0xffffffffu, act);
                if (act) peers = __match_any_sync(am, col);
                const uint32_t lead = act ? (uint32_t)__ffs((int)peers) - 1u : lane;
                const bool isLead = act && lead == lane;
                uint32_t h = (col * 2654435761u) >> 16 & (H - 1), id = 0;
                bool fresh = false;
                if (isLead)
                    for (;; h = (h + 1) & (H - 1)) { // at most CAP of the H places are taken
                        const uint32_t key = T.key[h];
                        if (key == col) {
                            id = T.idx[h];
                            break;
                        }
                        if (key == kFree) {
                            fresh = true;
                            break;
                        }
                    }
                __syncwarp();
                const uint32_t nm = __ballot_sync(0xffffffffu, fresh);
                if (fresh) {
                    id = cnt + (uint32_t)__popc(nm & below);
                    while (atomicCAS(&T.key[h], kFree, col) != kFree) h = (h + 1) & (H - 1);
                    T.idx[h] = (uint16_t)id;
                    T.slot[id] = (uint16_t)h;
                    T.col[id] = col;
                    T.acc[id] = 0.0;
                }
                cnt += (uint32_t)__popc(nm);
                __syncwarp();
                id = __shfl_sync(0xffffffffu, id, (int)lead);
                const uint32_t rank = (uint32_t)__popc(peers & below);
                const uint32_t rounds = __reduce_max_sync(0xffffffffu, (uint32_t)__popc(peers));
                for (uint32_t r = 0; r < rounds; ++r) {
                    if (act && rank == r) T.acc[id] = __dadd_rn(T.acc[id], prod);
                    __syncwarp();
                }
            }
        }
        for (uint32_t q = lane; q < cnt; q += 32) {
            ocol[(size_t)base + q] = T.col[q];
            osum[(size_t)base + q] = T.acc[q];
            T.key[T.slot[q]] = kFree;
        }
        if (lane == 0) nout[i] = cnt;
        __syncwarp();
    }
}

// Row i's nout entries from its candidates' place to its place in C, 8 lanes per row.
__global__ void __launch_bounds__(256) k_mult_pack(uint32_t n, const uint32_t* __restrict__ coff,
                                                   const uint32_t* __restrict__ crp,
                                                   const uint32_t* __restrict__ ocol,
                                                   const double* __restrict__ osum,
                                                   uint32_t* __restrict__ cci,
                                                   double* __restrict__ cva)
{
    const uint32_t lane = threadIdx.x & 7u;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; i < n;
         i += ((size_t)gridDim.x * blockDim.x) >> 3) {
        const uint32_t b = crp[i], len = crp[i + 1] - b;
        const size_t src = coff[i];
        for (uint32_t q = lane; q < len; q += 8) {
            cci[b + q] = ocol[src + q];
            cva[b + q] = osum[src + q];
        }
    }
}

// keys (column << 32 | position in the row's loop order) and the rounded products
__global__ void k_mult_expand(uint32_t n, const uint32_t* __restrict__ lrp,
                              const uint32_t* __restrict__ lci, const double* __restrict__ lva,
                              const uint32_t* __restrict__ rrp, const uint32_t* __restrict__ rci,
                              const double* __restrict__ rva, const uint32_t* __restrict__ coff,
                              uint64_t* __restrict__ keys, double* __restrict__ prod)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        uint32_t p = 0;
        const size_t base = coff[i];
        for (uint32_t k = lrp[i]; k < lrp[i + 1]; ++k) {
            const uint32_t j = lci[k];
            const double a = lva[k];
            for (uint32_t l = rrp[j]; l < rrp[j + 1]; ++l, ++p) {
                keys[base + p] = (uint64_t)rci[l] << 32 | p;
                prod[base + p] = a * rva[l];
            }
        }
    }
}

// distinct columns per row (the keys of each row sorted)
__global__ void k_mult_distinct(uint32_t n, const uint32_t* __restrict__ coff,
                                const uint64_t* __restrict__ keys, uint32_t* __restrict__ nout)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        uint32_t d = 0;
        for (uint32_t q = coff[i]; q < coff[i + 1]; ++q)
            if (q == coff[i] || (keys[q] >> 32) != (keys[q - 1] >> 32)) ++d;
        nout[i] = d;
    }
}

// one entry per distinct column: its sum in loop order, its column, and the key
// first position << 32 | group index that orders the row as MAT::Mult does
__global__ void k_mult_groups(uint32_t n, const uint32_t* __restrict__ coff,
                              const uint64_t* __restrict__ keys, const double* __restrict__ prod,
                              const uint32_t* __restrict__ crp, uint64_t* __restrict__ okeys,
                              uint32_t* __restrict__ gcol, double* __restrict__ gsum)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t b = coff[i], e = coff[i + 1];
        uint32_t g = 0;
        for (uint32_t q = b; q < e;) {
            const uint32_t col = (uint32_t)(keys[q] >> 32);
            const uint32_t first = (uint32_t)keys[q];
            double s = 0.0;
            for (; q < e && (uint32_t)(keys[q] >> 32) == col; ++q)
                s = __dadd_rn(s, prod[(size_t)b + (uint32_t)keys[q]]);
            const size_t o = (size_t)crp[i] + g;
            okeys[o] = (uint64_t)first << 32 | g;
            gcol[o] = col;
            gsum[o] = s;
            ++g;
        }
    }
}

__global__ void k_mult_out(uint32_t n, const uint32_t* __restrict__ crp,
                           const uint64_t* __restrict__ okeys, const uint32_t* __restrict__ gcol,
                           const double* __restrict__ gsum, uint32_t* __restrict__ cci,
                           double* __restrict__ cva)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        for (uint32_t q = crp[i]; q < crp[i + 1]; ++q) {
            const size_t src = (size_t)crp[i] + (uint32_t)okeys[q];
            cci[q] = gcol[src];
            cva[q] = gsum[src];
        }
}

} // namespace

namespace {

template <uint32_t CAP, int WARPS>
int launch_hash(Ctx& c, const Mat& L, const Mat& R, uint32_t lo, const uint32_t* coff,
                uint32_t* ocol, double* osum, uint32_t* nout)
{
    const auto kern = k_mult_hash<CAP, WARPS>;
    const size_t smem = WARPS * sizeof(HashRow<CAP>);
    FB_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    const int g = (int)std::max<size_t>(
        1, std::min<size_t>(((size_t)L.nrow + WARPS - 1) / WARPS,
                            (size_t)resident_grid(c, (const void*)kern, WARPS * 32, smem)));
    kern<<<g, WARPS * 32, smem, c.stream>>>(L.nrow, lo, L.rowPtr, L.colInd, L.val, R.rowPtr,
                                            R.colInd, R.val, coff, ocol, osum, nout);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

// Column order and sums by sorting: products with a row of more than kHashMost candidates.
int mult_sorted(Ctx& c, Tmp& t, const Mat& L, const Mat& R, uint32_t ncand, const uint32_t* coff,
                uint32_t* nout, uint32_t* tiles, Mat& T)
{
    cudaStream_t s = c.stream;
    const uint32_t n = L.nrow;
    const int g = grid_for(n, 256);
    int e;
    uint64_t *keys = nullptr, *okeys = nullptr;
    uint32_t* gcol = nullptr;
    double *prod = nullptr, *gsum = nullptr;
    if ((e = t.get(&keys, ncand)) || (e = t.get(&prod, ncand))) return e;
    k_mult_expand<<<g, 256, 0, s>>>(n, L.rowPtr, L.colInd, L.val, R.rowPtr, R.colInd, R.val,
                                    coff, keys, prod);
    FB_CUDA(cudaGetLastError());
    if ((e = sort_row_keys(c, t, n, coff, keys, ncand))) return e;
    k_mult_distinct<<<g, 256, 0, s>>>(n, coff, keys, nout);
    FB_CUDA(cudaGetLastError());
    if ((e = scan_counts(s, n, nout, T.rowPtr, tiles))) return e;
    FB_CUDA(cudaMemcpyAsync(&T.nnz, T.rowPtr + n, 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if ((e = t.get(&okeys, T.nnz)) || (e = t.get(&gcol, T.nnz)) || (e = t.get(&gsum, T.nnz)) ||
        (e = dmalloc((void**)&T.colInd, (size_t)T.nnz * 4, s)) ||
        (e = dmalloc((void**)&T.val, (size_t)T.nnz * 8, s)))
        return e;
    k_mult_groups<<<g, 256, 0, s>>>(n, coff, keys, prod, T.rowPtr, okeys, gcol, gsum);
    FB_CUDA(cudaGetLastError());
    if ((e = sort_row_keys(c, t, n, T.rowPtr, okeys, T.nnz))) return e;
    k_mult_out<<<g, 256, 0, s>>>(n, T.rowPtr, okeys, gcol, gsum, T.colInd, T.val);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

// The sizes, rowPtr, colInd and val of T = L R.
int mult_arrays(Ctx& c, const Mat& L, const Mat& R, Mat& T)
{
    cudaStream_t s = c.stream;
    const uint32_t n = L.nrow;
    Tmp t(s);
    int e;
    uint32_t *cnt = nullptr, *coff = nullptr, *tiles = nullptr;
    MultPlan* dplan = nullptr;
    if ((e = t.get(&cnt, n)) || (e = t.get(&coff, (size_t)n + 1)) ||
        (e = t.get(&tiles, (n + (size_t)kTile - 1) / kTile)) || (e = t.get(&dplan, 1)) ||
        (e = dmalloc((void**)&T.rowPtr, ((size_t)n + 1) * 4, s)))
        return e;
    FB_CUDA(cudaMemsetAsync(dplan, 0, sizeof(MultPlan), s));
    k_mult_count<<<grid_for(n, 256), 256, 0, s>>>(n, L.rowPtr, L.colInd, R.rowPtr, cnt, dplan);
    FB_CUDA(cudaGetLastError());
    if ((e = scan_counts(s, n, cnt, coff, tiles))) return e;
    MultPlan plan;
    FB_CUDA(cudaMemcpyAsync(&plan, dplan, sizeof(plan), cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if (plan.total == 0) return kErrMatSize; // MAT::Mult would build a matrix with no entries
    if (plan.total > 0xffffffffull) return kErrMatSize;
    const uint32_t ncand = (uint32_t)plan.total;
    T.nrow = n;
    T.mcol = R.mcol;
    if (plan.has[3]) return mult_sorted(c, t, L, R, ncand, coff, cnt, tiles, T);
    uint32_t* ocol = nullptr;
    double* osum = nullptr;
    if ((e = t.get(&ocol, ncand)) || (e = t.get(&osum, ncand))) return e;
    if ((plan.has[0] && (e = launch_hash<kHashCap0, 8>(c, L, R, 0, coff, ocol, osum, cnt))) ||
        (plan.has[1] &&
         (e = launch_hash<kHashCap1, 8>(c, L, R, kHashCap0, coff, ocol, osum, cnt))) ||
        (plan.has[2] &&
         (e = launch_hash<kHashMost, 4>(c, L, R, kHashCap1, coff, ocol, osum, cnt))))
        return e;
    if ((e = scan_counts(s, n, cnt, T.rowPtr, tiles))) return e;
    FB_CUDA(cudaMemcpyAsync(&T.nnz, T.rowPtr + n, 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if ((e = dmalloc((void**)&T.colInd, (size_t)T.nnz * 4, s)) ||
        (e = dmalloc((void**)&T.val, (size_t)T.nnz * 8, s)))
        return e;
    k_mult_pack<<<grid_for((size_t)n * 8, 256), 256, 0, s>>>(n, coff, T.rowPtr, ocol, osum, T.colInd,
                                                             T.val);
    FB_CUDA(cudaGetLastError());
    return kOk;
}

} // namespace

int m_mult(Ctx& c, const Mat& L, const Mat& R, Mat& C)
{
    if (L.grid || R.grid || !L.val || !R.val) return kErrInputPar; // stored values needed
    if (L.mcol != R.nrow) return kErrNonmatch;
    if (L.nrow == 0 || R.mcol == 0) return kErrMatSize;
    Mat T;
    const int e = mult_arrays(c, L, R, T);
    if (e) {
        cudaStreamSynchronize(c.stream);
        m_free(T);
        return e;
    }
    return m_adopt(C, T, c.stream);
}

namespace {

// ---- MAT::Add (src/MAT.cxx:652-713): C = a A + b B -------------------------------------------
// Row i of C: A's entries in order as a A(i,k); then each entry of B's row in order is added
// to the first entry of A's row with its column -- or to the first of B's entries already
// appended to this row, the one extra slot MAT::Add's search window reaches -- else appended
// as b B(i,k); finally each row sorted by column, stably (SortCSRRow). Products and sums are
// rounded separately as the reference rounds them.

__global__ void k_add_rows(uint32_t n, double a, double b, const uint32_t* __restrict__ arp,
                           const uint32_t* __restrict__ aci, const double* __restrict__ ava,
                           const uint32_t* __restrict__ brp, const uint32_t* __restrict__ bci,
                           const double* __restrict__ bva, uint32_t* __restrict__ tci,
                           double* __restrict__ tva, uint32_t* __restrict__ nout)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t base = (size_t)arp[i] + brp[i];
        const uint32_t c1 = arp[i + 1] - arp[i];
        uint32_t cnt = 0;
        for (uint32_t k = arp[i]; k < arp[i + 1]; ++k, ++cnt) {
            tci[base + cnt] = aci[k];
            tva[base + cnt] = __dmul_rn(a, ava[k]);
        }
        for (uint32_t k = brp[i]; k < brp[i + 1]; ++k) {
            const uint32_t col = bci[k];
            const double v = __dmul_rn(b, bva[k]);
            const uint32_t window = cnt > c1 ? c1 + 1 : c1;
            uint32_t l = 0;
            for (; l < window; ++l)
                if (tci[base + l] == col) break;
            if (l < window) {
                tva[base + l] = __dadd_rn(tva[base + l], v);
            } else {
                tci[base + cnt] = col;
                tva[base + cnt] = v;
                ++cnt;
            }
        }
        nout[i] = cnt;
    }
}

__global__ void k_add_keys(uint32_t n, const uint32_t* __restrict__ arp,
                           const uint32_t* __restrict__ brp, const uint32_t* __restrict__ crp,
                           const uint32_t* __restrict__ tci, uint64_t* __restrict__ keys)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t base = (size_t)arp[i] + brp[i];
        for (uint32_t q = crp[i]; q < crp[i + 1]; ++q) {
            const uint32_t p = q - crp[i];
            keys[q] = (uint64_t)tci[base + p] << 32 | p;
        }
    }
}

__global__ void k_add_out(uint32_t n, const uint32_t* __restrict__ arp,
                          const uint32_t* __restrict__ brp, const uint32_t* __restrict__ crp,
                          const uint64_t* __restrict__ keys, const double* __restrict__ tva,
                          uint32_t* __restrict__ cci, double* __restrict__ cva)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t base = (size_t)arp[i] + brp[i];
        for (uint32_t q = crp[i]; q < crp[i + 1]; ++q) {
            cci[q] = (uint32_t)(keys[q] >> 32);
            cva[q] = tva[base + (uint32_t)keys[q]];
        }
    }
}

} // namespace

int m_add(Ctx& c, double a, const Mat& A, double b, const Mat& B, Mat& C)
{
    if (A.grid || B.grid || !A.val || !B.val) return kErrInputPar;
    if (A.nrow != B.nrow || A.mcol != B.mcol) return kErrNonmatch;
    const uint64_t cap = (uint64_t)A.nnz + B.nnz;
    if (cap > 0xffffffffull) return kErrMatSize;
    cudaStream_t s = c.stream;
    const uint32_t n = A.nrow;
    Tmp t(s);
    int e;
    uint32_t *tci = nullptr, *nout = nullptr, *crp = nullptr, *tiles = nullptr, *cci = nullptr;
    double *tva = nullptr, *cva = nullptr;
    uint64_t* keys = nullptr;
    if ((e = t.get(&tci, cap)) || (e = t.get(&tva, cap)) || (e = t.get(&nout, n)) ||
        (e = t.get(&crp, (size_t)n + 1)) || (e = t.get(&tiles, (n + (size_t)kTile - 1) / kTile)))
        return e;
    const int g = grid_for(n, 256);
    k_add_rows<<<g, 256, 0, s>>>(n, a, b, A.rowPtr, A.colInd, A.val, B.rowPtr, B.colInd, B.val,
                                 tci, tva, nout);
    FB_CUDA(cudaGetLastError());
    if ((e = scan_counts(s, n, nout, crp, tiles))) return e;
    uint32_t nnzC = 0;
    FB_CUDA(cudaMemcpyAsync(&nnzC, crp + n, 4, cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
    if ((e = t.get(&keys, nnzC)) || (e = t.get(&cci, nnzC)) || (e = t.get(&cva, nnzC))) return e;
    k_add_keys<<<g, 256, 0, s>>>(n, A.rowPtr, B.rowPtr, crp, tci, keys);
    FB_CUDA(cudaGetLastError());
    if ((e = sort_row_keys(c, t, n, crp, keys, nnzC))) return e;
    k_add_out<<<g, 256, 0, s>>>(n, A.rowPtr, B.rowPtr, crp, keys, tva, cci, cva);
    FB_CUDA(cudaGetLastError());
    FB_CUDA(cudaStreamSynchronize(s));
    return m_upload(C, n, A.mcol, nnzC, crp, cci, cva, false, s);
}

} // namespace fb
