// batch_resident.cuh -- batched Jacobi-PCG with a system's vectors on chip.
//
// One thread-block cluster of 1, 2, 4 or 8 blocks takes one system with all its right-hand
// sides. Block b of the cluster owns a contiguous range of its rows and keeps p, q and r of
// those rows in shared memory, x in registers; a gathered p of another block's row comes
// through distributed shared memory. Only the matrix, the Jacobi weights and the row lengths are
// read each iteration, once for all right-hand sides. The matrix is stored for it at creation
// in slices of 32 rows, entry k of a slice's rows side by side (coalesced; a row's entries in
// CSR order), with 16-bit columns relative to the system.
//
// Why: with the vectors in global memory (batch_pcg) an iteration gathered z and p_old of
// every entry per right-hand side and moved 424 bytes per row and iteration for four of them
// (FP64), and one block of 256 threads took a 16,384-row system: on a batch of 512 systems the
// longest-running one, alone on an eighth of an SM, was the batch's time. Measured on B200, 512
// shifted 2D Poisson systems of 16^2 to 128^2 rows with four right-hand sides: 72.7 -> 9.8 ms (FP64),
// 67.0 -> 8.8 ms (FP32 with reliable updates); one right-hand side 22.5 -> 5.9 ms. An iteration
// of a 16,384-row system on 8 SMs takes about 10 us, 39% of issue slots busy: shared-memory
// traffic and the three cluster barriers share the rest. Loading the next entries before
// gathering the current ones measured slower (10.5 ms, spills). Rows, right-hand
// sides and operations are those of batch_pcg and batch_pcg_rel: only the order of the FP64
// partial sums differs, and FP32 vectors see the same operations in the same order.
#pragma once

#include "internal.h"

namespace fb {

// Everything a launch needs; T is the iteration's precision.
template <typename T>
struct ResArgs {
    uint32_t        items, first; // systems of this class: order[first .. first + items)
    uint32_t        nrhs, N;
    const uint32_t* sysRow;
    const uint32_t* order;
    const uint32_t* sliceBase; // a system's first slice
    const uint32_t* sliceOff;  // a slice's first entry / 32
    const uint16_t* rowLen;
    const uint16_t* col;
    const T*        val;
    const T*        dinv;
    const T*        b; // rhs-major [nrhs][N]
    T*              x;
    uint32_t*       iters;
    double*         resRel;
    double          relTol;
    uint32_t        maxIter;
    unsigned*       queue;
    // reliable updates (FP32 iterations)
    const double* val64;
    const double* b64;
    double*       x64;
    double        delta;
};

// Values per thread and array: three FP64 arrays of a 1,024-thread block take 196,608 bytes.
// FP32 takes as many: 16 would fit, but a system then runs on half the SMs, and the 512-system
// batch took 11.0 instead of 8.8 ms.
constexpr int kResVals = 8;

// NR values of one row, moved in pieces of at most 16 bytes. Piece i of row r lies at
// ((i * CAP) + r) * 16 bytes of its array, so a warp's rows are side by side.
template <typename T, int NR>
struct ResPack {
    static constexpr int W = NR * (int)sizeof(T) >= 16 ? 16 / (int)sizeof(T) : NR; // values a piece
    static constexpr int PIECES = NR / W;
};

__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void ld_piece(uint32_t a, double (&v)[2])
{
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_piece(uint32_t a, double (&v)[1])
{
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[0]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_piece(uint32_t a, float (&v)[4])
{
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_piece(uint32_t a, float (&v)[2])
{
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_piece(uint32_t a, float (&v)[1])
{
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[0]) : "r"(a) : "memory");
}
template <typename T, int W>
struct alignas(W * sizeof(T)) ResPiece {
    T v[W];
};

// The sum over the warp of each of NV (a power of two) values: lanes exchange halves of the
// values, so NV values cost NV - 1 + 5 - log2(NV) exchanges instead of 5 NV. Every lane returns
// value lane * NV / 32; the order of the additions is fixed.
template <int NV>
__device__ __forceinline__ double warp_sum_each(double (&v)[NV])
{
    const uint32_t lane = threadIdx.x & 31u;
    int o = 16;
#pragma unroll
    for (int half = NV / 2; half > 0; half >>= 1, o >>= 1) {
        const bool up = (lane & (uint32_t)o) != 0;
#pragma unroll
        for (int j = 0; j < NV / 2; ++j)
            if (j < half) {
                const double keep = up ? v[j + half] : v[j], send = up ? v[j] : v[j + half];
                v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    double s = v[0];
    for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Every thread of the cluster (of the block, for a cluster of one).
__device__ __forceinline__ void cluster_meet(uint32_t cs)
{
    __syncwarp(); // the cluster barrier takes whole warps
    if (cs > 1)
        asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                     "barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
        __syncthreads();
}

template <typename T, int NR, int TH, bool REL>
__global__ void __launch_bounds__(TH, 1024 / TH) batch_resident(ResArgs<T> a)
{
    constexpr int RPT = kResVals / NR; // rows a thread owns
    constexpr uint32_t CAP = (uint32_t)TH * RPT;
    constexpr int W = ResPack<T, NR>::W, PIECES = ResPack<T, NR>::PIECES;
    constexpr int NWARP = TH / 32, NVMAX = 4 * NR;
    // one right-hand side's scalars, the same in every block of the cluster
    struct Rhs {
        double   rz, rzold, beta, rmax, res, tol, last, true0, prev, sc;
        T        alpha;
        int      active, fresh, stall, trig;
        unsigned its;
    };
    extern __shared__ __align__(16) unsigned char resident[];
    __shared__ Rhs st[NR];
    __shared__ double wsum[NWARP][NVMAX];
    __shared__ double slot[2][8][NVMAX]; // the blocks' sums, by turn
    __shared__ double tot[NVMAX];
    __shared__ unsigned item;
    __shared__ int nact, refresh;
    uint32_t cs, rank;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(cs));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    uint32_t turn = 0;
    pdl_release(); // the next size class may move in as blocks of this one leave

    // row lr of this block's array A, and of another block's p
    using Piece = ResPiece<T, W>;
    Piece* const P = reinterpret_cast<Piece*>(resident);
    Piece* const Q = P + CAP * PIECES;
    Piece* const R = Q + CAP * PIECES;
    auto load = [&](const Piece* A, uint32_t lr, T (&v)[NR]) {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const Piece t = A[i * CAP + lr];
#pragma unroll
            for (int j = 0; j < W; ++j) v[i * W + j] = t.v[j];
        }
    };
    auto load_far = [&](uint32_t own, uint32_t lr, T (&v)[NR]) {
        const uint32_t at = mapa_u32(smem_addr(P), own);
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            T t[W];
            ld_piece(at + (i * CAP + lr) * (uint32_t)sizeof(Piece), t);
#pragma unroll
            for (int j = 0; j < W; ++j) v[i * W + j] = t[j];
        }
    };
    auto store = [&](Piece* A, uint32_t lr, const T (&v)[NR]) {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            Piece t;
#pragma unroll
            for (int j = 0; j < W; ++j) t.v[j] = v[i * W + j];
            A[i * CAP + lr] = t;
        }
    };
    // tot[k] = the cluster's sum of v[k], for warp 0's step(); then a block barrier
    auto reduce = [&](auto& v, auto step) {
        constexpr int NV = (int)(sizeof(v) / sizeof(double));
        const double w = warp_sum_each<NV>(v);
        if (lane % (32 / NV) == 0) wsum[wid][lane / (32 / NV)] = w;
        __syncthreads();
        double s = 0.0;
        if (wid == 0) { // 32 / NV lanes per value, then their sum in lane < NV
            constexpr int G = 32 / NV, PER = (NWARP + G - 1) / G;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int w = (int)(lane / NV) * PER + k;
                if (w < NWARP) s += wsum[w][lane % NV];
            }
#pragma unroll
            for (int o = 16; o >= NV; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (cs > 1 && lane < NV) {
                const uint32_t mine = smem_addr(&slot[turn & 1][rank][lane]);
                for (uint32_t r = 0; r < cs; ++r)
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(mapa_u32(mine, r)), "d"(s)
                                 : "memory");
            }
        }
        if (cs > 1) cluster_meet(cs);
        if (wid == 0) {
            if (lane < NV) {
                if (cs > 1) {
                    s = 0.0;
                    for (uint32_t r = 0; r < cs; ++r) s += slot[turn & 1][r][lane];
                }
                tot[lane] = s;
            }
            __syncwarp();
            step();
        }
        ++turn;
        __syncthreads();
    };

    for (;;) {
        cluster_meet(cs); // nobody still uses the previous system's state
        if (rank == 0 && tid == 0) {
            const unsigned it = atomicAdd(a.queue, 1u);
            for (uint32_t r = 0; r < cs; ++r)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_u32(smem_addr(&item), r)),
                             "r"(it)
                             : "memory");
        }
        cluster_meet(cs);
        if (item >= a.items) break;
        const uint32_t sys = a.order[a.first + item];
        const uint32_t s0 = a.sysRow[sys], n = a.sysRow[sys + 1] - s0;
        const uint32_t rpc = ((n + cs - 1) / cs + 31u) & ~31u; // rows per block, whole slices
        const uint32_t magic = (uint32_t)((1ull << 32) / rpc) + 1u; // c / rpc for c < 65,536
        const uint32_t base = rank * rpc;
        const uint32_t rows = n > base ? (n - base < rpc ? n - base : rpc) : 0u;
        const size_t g0 = (size_t)s0 + base;
        const uint32_t sl0 = a.sliceBase[sys] + base / 32;
        T x[RPT][NR];
        auto dinv = [&](uint32_t lr) { return a.dinv[g0 + lr]; };

        // the scale of the FP32 iterations: ||b||
        if constexpr (REL) {
            double bb[NR];
#pragma unroll
            for (int k = 0; k < NR; ++k) bb[k] = 0.0;
            for (uint32_t lr = tid; lr < rows; lr += TH)
#pragma unroll
                for (int k = 0; k < NR; ++k) {
                    if (k >= (int)a.nrhs) break;
                    const double bi = a.b64[(size_t)k * a.N + g0 + lr];
                    a.x64[(size_t)k * a.N + g0 + lr] = 0.0;
                    bb[k] = fma(bi, bi, bb[k]);
                }
            reduce(bb, [&] {
                if (lane < NR) {
                    Rhs& h = st[lane];
                    const double nb = sqrt(tot[lane]);
                    h.true0 = h.prev = nb;
                    h.sc = nb > 0.0 ? nb : 1.0;
                    h.active = nb > 0.0;
                    h.stall = 0;
                }
            });
        }
        // start: x = 0, r = b, z = diagInv .* r, p = z; (r, r), (z, r)
        {
            double acc[2 * NR];
#pragma unroll
            for (int k = 0; k < 2 * NR; ++k) acc[k] = 0.0;
#pragma unroll
            for (int j = 0; j < RPT; ++j)
#pragma unroll
                for (int k = 0; k < NR; ++k) x[j][k] = T(0);
#pragma unroll
            for (int j = 0; j < RPT; ++j) {
                const uint32_t lr = tid + (uint32_t)j * TH;
                if (lr >= rows) break;
                const T dj = dinv(lr);
                T r[NR], z[NR];
#pragma unroll
                for (int k = 0; k < NR; ++k) {
                    r[k] = T(0);
                    if (k < (int)a.nrhs) {
                        const size_t o = (size_t)k * a.N + g0 + lr;
                        if constexpr (REL)
                            r[k] = (T)(a.b64[o] / st[k].sc);
                        else
                            r[k] = a.b[o];
                    }
                    z[k] = dj * r[k];
                    acc[k] += (double)r[k] * r[k];
                    acc[NR + k] += (double)z[k] * r[k];
                }
                store(R, lr, r);
                store(P, lr, z);
            }
            reduce(acc, [&] {
                int act = 0;
                if (lane < NR) {
                    Rhs& h = st[lane];
                    h.res = sqrt(tot[lane]);
                    h.rz = tot[NR + lane];
                    h.rmax = h.res;
                    h.beta = 0.0;
                    h.fresh = 1; // the next p is z (first iteration, or after a restart)
                    h.its = 0;
                    h.last = 1.0;
                    if constexpr (!REL) {
                        h.tol = a.relTol * h.res;
                        h.active = h.res > h.tol && tot[lane] > 0.0;
                    }
                    act = h.active;
                }
                const uint32_t m = __ballot_sync(0xffffffffu, act != 0);
                if (lane == 0) nact = __popc(m);
            });
        }
        uint32_t it = 0;
        while (nact > 0 && it < a.maxIter) {
            ++it;
            bool act[NR];
#pragma unroll
            for (int k = 0; k < NR; ++k) act[k] = st[k].active != 0;
            // p = z + beta p_old (or z)
            {
                T beta[NR];
                bool fresh[NR];
#pragma unroll
                for (int k = 0; k < NR; ++k) {
                    beta[k] = (T)st[k].beta;
                    fresh[k] = st[k].fresh != 0;
                }
#pragma unroll
                for (int j = 0; j < RPT; ++j) {
                    const uint32_t lr = tid + (uint32_t)j * TH;
                    if (lr >= rows) break;
                    const T dj = dinv(lr);
                    T p[NR], r[NR];
                    load(P, lr, p);
                    load(R, lr, r);
#pragma unroll
                    for (int k = 0; k < NR; ++k)
                        if (act[k]) {
                            const T z = dj * r[k];
                            p[k] = fresh[k] ? z : fma(beta[k], p[k], z);
                        }
                    store(P, lr, p);
                }
            }
            cluster_meet(cs); // every block's p is in place
            // q = A p; (q, p)
            {
                double pq[NR];
#pragma unroll
                for (int k = 0; k < NR; ++k) pq[k] = 0.0;
                for (uint32_t lr = tid; lr - lane < rows; lr += TH) {
                    const uint32_t len = lr < rows ? a.rowLen[g0 + lr] : 0u;
                    const uint32_t wide = __reduce_max_sync(0xffffffffu, len);
                    const size_t e0 = (size_t)a.sliceOff[sl0 + lr / 32] * 32 + lane;
                    T s[NR];
#pragma unroll
                    for (int k = 0; k < NR; ++k) s[k] = T(0);
                    for (uint32_t k0 = 0; k0 < wide; k0 += 4) {
                        uint32_t c[4];
                        T v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const bool in = k0 + u < len;
                            c[u] = in ? __ldg(a.col + e0 + (size_t)(k0 + u) * 32) : 0u;
                            v[u] = in ? __ldg(a.val + e0 + (size_t)(k0 + u) * 32) : T(0);
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (k0 + u >= len) continue;
                            const uint32_t lc = c[u] - base;
                            T p[NR];
                            if (lc < rpc) {
                                load(P, lc, p);
                            } else { // another block's row
                                const uint32_t own = __umulhi(c[u], magic);
                                load_far(own, c[u] - own * rpc, p);
                            }
#pragma unroll
                            for (int k = 0; k < NR; ++k) s[k] = fma(v[u], p[k], s[k]);
                        }
                    }
                    if (lr < rows) {
                        T p[NR];
                        load(P, lr, p);
                        store(Q, lr, s);
#pragma unroll
                        for (int k = 0; k < NR; ++k) pq[k] += (double)s[k] * p[k];
                    }
                }
                reduce(pq, [&] {
                    if (lane < NR) {
                        Rhs& h = st[lane];
                        h.alpha = h.active && tot[lane] != 0.0 ? (T)(h.rz / tot[lane]) : T(0);
                        h.fresh = 0;
                    }
                });
            }
            // x += alpha p, r -= alpha q, z = diagInv .* r; (r, r), (z, r)
            {
                double acc[2 * NR];
#pragma unroll
                for (int k = 0; k < 2 * NR; ++k) acc[k] = 0.0;
                T alpha[NR];
#pragma unroll
                for (int k = 0; k < NR; ++k) alpha[k] = st[k].alpha;
#pragma unroll
                for (int j = 0; j < RPT; ++j) {
                    const uint32_t lr = tid + (uint32_t)j * TH;
                    if (lr < rows) {
                        const T dj = dinv(lr);
                        T p[NR], q[NR], r[NR];
                        load(P, lr, p);
                        load(Q, lr, q);
                        load(R, lr, r);
#pragma unroll
                        for (int k = 0; k < NR; ++k)
                            if (act[k]) {
                                x[j][k] = fma(alpha[k], p[k], x[j][k]);
                                r[k] = fma(-alpha[k], q[k], r[k]);
                                const T z = dj * r[k];
                                acc[k] += (double)r[k] * r[k];
                                acc[NR + k] += (double)z * r[k];
                            }
                        store(R, lr, r);
                    }
                }
                reduce(acc, [&] {
                    int on = 0, rf = 0;
                    if (lane < NR && st[lane].active) {
                        Rhs& h = st[lane];
                        const double rr = tot[lane], zr = tot[NR + lane], res = sqrt(rr);
                        h.res = h.last = res;
                        if constexpr (REL) {
                            h.trig = 0;
                            if (res > h.rmax) h.rmax = res;
                            h.rzold = h.rz;
                            if (res < a.relTol || res < a.delta * h.rmax || !(rr == rr)) {
                                h.trig = rf = 1;
                            } else {
                                h.beta = zr / h.rz;
                                h.rz = zr;
                            }
                        } else if (res < h.tol || !(zr == zr)) {
                            h.active = 0;
                            h.its = it;
                        } else {
                            h.beta = zr / h.rz;
                            h.rz = zr;
                        }
                        on = h.active;
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, on != 0);
                    const uint32_t f = __ballot_sync(0xffffffffu, rf != 0);
                    if (lane == 0) {
                        nact = __popc(m);
                        refresh = f != 0;
                    }
                });
            }
            if constexpr (REL) {
                if (!refresh) continue; // the same in every block
                // 1. x64 += s x32, x32 = 0
#pragma unroll
                for (int j = 0; j < RPT; ++j) {
                    const uint32_t lr = tid + (uint32_t)j * TH;
                    if (lr < rows)
#pragma unroll
                        for (int k = 0; k < NR; ++k)
                            if (act[k]) {
                                double& xo = a.x64[(size_t)k * a.N + g0 + lr];
                                xo = fma(st[k].sc, (double)x[j][k], xo);
                                x[j][k] = T(0);
                            }
                }
                cluster_meet(cs);
                // 2. r = b - A x64 in FP64; r32 = r / s; z32 = diagInv .* r32
                double rr[4 * NR];
#pragma unroll
                for (int k = 0; k < 4 * NR; ++k) rr[k] = 0.0;
#pragma unroll
                for (int j = 0; j < RPT; ++j) {
                    const uint32_t lr = tid + (uint32_t)j * TH;
                    if (lr >= rows) break;
                    const T dj = dinv(lr);
                    const uint32_t len = a.rowLen[g0 + lr];
                    const size_t e0 = (size_t)a.sliceOff[sl0 + lr / 32] * 32 + lane;
                    double sum[NR];
#pragma unroll
                    for (int k = 0; k < NR; ++k) sum[k] = 0.0;
                    for (uint32_t q = 0; q < len; ++q) {
                        const double v = __ldg(a.val64 + e0 + (size_t)q * 32);
                        const size_t o = (size_t)s0 + __ldg(a.col + e0 + (size_t)q * 32);
#pragma unroll
                        for (int k = 0; k < NR; ++k) // other blocks' x64 come from L2
                            if (act[k])
                                sum[k] = fma(v, __ldcg(a.x64 + (size_t)k * a.N + o), sum[k]);
                    }
                    T r[NR];
                    load(R, lr, r);
#pragma unroll
                    for (int k = 0; k < NR; ++k)
                        if (act[k]) {
                            const double ri = a.b64[(size_t)k * a.N + g0 + lr] - sum[k];
                            r[k] = (T)(ri / st[k].sc);
                            const T z = dj * r[k];
                            rr[k] = fma(ri, ri, rr[k]);
                            rr[NR + k] += (double)r[k] * r[k];
                            rr[2 * NR + k] += (double)z * r[k];
                        }
                    store(R, lr, r);
                }
                reduce(rr, [&] {
                    int on = 0;
                    if (lane < NR && st[lane].active) {
                        Rhs& h = st[lane];
                        const double tr = sqrt(tot[lane]);
                        // three refreshes of its own in a row gaining less than sqrt(delta):
                        // the tolerance is below what the FP32 iterations attain here (a
                        // refresh another right-hand side asked for is not counted)
                        if (h.trig) {
                            h.stall = tr > sqrt(a.delta) * h.prev ? h.stall + 1 : 0;
                            h.prev = tr;
                        }
                        if (tr < a.relTol * h.true0 || !(tr == tr) || h.stall >= 3) {
                            h.active = 0;
                            h.its = it;
                            h.res = tr / h.sc;
                        } else {
                            const double rs = sqrt(tot[NR + lane]);
                            // a refreshed residual far above the recursive one: p = z
                            if (rs > 4.0 * h.res) h.fresh = 1;
                            // beta from the refreshed residual and the (z, r) of the previous
                            // iteration
                            h.beta = tot[2 * NR + lane] / h.rzold;
                            h.rz = tot[2 * NR + lane];
                            h.rmax = rs;
                            h.res = rs;
                        }
                        on = h.active;
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, on != 0);
                    if (lane == 0) nact = __popc(m);
                });
            }
        }
        // the solution; with reliable updates only what is still in FP32 (maxIter reached)
#pragma unroll
        for (int j = 0; j < RPT; ++j) {
            const uint32_t lr = tid + (uint32_t)j * TH;
            if (lr < rows)
#pragma unroll
                for (int k = 0; k < NR; ++k) {
                    if (k >= (int)a.nrhs) break;
                    const size_t o = (size_t)k * a.N + g0 + lr;
                    if constexpr (REL) {
                        if (st[k].active) a.x64[o] = fma(st[k].sc, (double)x[j][k], a.x64[o]);
                    } else {
                        a.x[o] = x[j][k];
                    }
                }
        }
        if (rank == 0 && tid < a.nrhs) {
            const Rhs& h = st[tid];
            const size_t o = (size_t)sys * a.nrhs + tid;
            a.iters[o] += h.active ? it : h.its;
            if constexpr (REL)
                a.resRel[o] = h.true0 > 0 ? h.res * h.sc / h.true0 : 0.0;
            else
                a.resRel[o] = h.tol > 0 ? h.last * a.relTol / h.tol : 0.0;
        }
    }
    pdl_wait(); // a later class ends after the earlier ones have
}

} // namespace fb
