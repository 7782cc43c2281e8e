// plane_walk.cuh -- rows of 3D seven-point stencil masks, walked plane by plane.
#pragma once

#include "internal.h"

namespace fb {

// A row kernel whose operand is formed from several vectors gathers each of them seven times a
// row: +-1 mostly hit L1, +-S1 and +-S2 come from L2, 3.8 loads a row and vector, and that
// traffic bounds it. Here a block walks `chunk` consecutive planes (S2 rows each) over
// kWalkCols * kBlock columns: the values of a plane's columns and of the S1 columns on both
// sides are formed once, by coalesced loads two planes ahead, and shared; the planes below and
// above are the thread's own columns, in registers. A row's products are summed in the order of
// its offsets, as row_apply does (the same bits). Any S1 <= kWalkS1 and S2, aligned or not.
// FP64 CG: see cg_spmv_walk. FP64 BiCGStab, three vectors and two: 57 to 47 us an iteration at
// 101^3, 51 to 47 at 100^3 and 168 to 129 at 150^3 (against 16-byte groups). Operands of one vector gain nothing: products
// at 127^3 14.4 us both ways, at 128^3 14.8 against the 10.3 of 16-byte groups.
constexpr uint32_t kWalkS1 = kBlock; // 2 S1 edge values a plane, two a thread
constexpr int kWalkCols = 2;         // columns a thread (1: 50 us at 101^3, 139 at 150^3)
// Planes an item walks at least; it loads two more. From three on both engines gain: BiCGStab 44 to
// 40 us an iteration at 90^3, FP64 CG solves 6.5 to 5.6, 5.6 to 5.2 and 5.0 to 4.8 ms at 95^3, 90^3
// and 85^3. Below, some sizes gain and their neighbours lose, the other kernels and the walk, us an
// iteration: FP64 CG 80^3 18.7 and 18.2, 72^3 17.2 and 17.9, 64^3 16.3 and 15.7, 56^3 14.7 and 14.9,
// 47^3 13.0 and 13.5, 24^3 11.6 and 12.1; BiCGStab 72^3 27.3 and 25.1, 64^3 23.1 and 24.6, 56^3 22.2
// and 21.3, 50^3 20.1 and 21.2.
constexpr uint32_t kWalkChunk = 3;

struct PlaneWalk {
    uint32_t tiles = 0; // blocks' items: segs column segments x chunks of planes; 0: not in use
    uint32_t segs = 0, chunk = 0, planes = 0;
};

template <typename T>
inline size_t walk_smem(const CSRView<T>& A)
{
    return 3 * sizeof(T) * ((size_t)kWalkCols * kBlock + 2 * A.udelta[5]);
}

// load(row) gives the operands of a row's value (out of range: not called), form(operands) the
// value, own(row, value, sum) consumes a row. RAW is load's result.
template <typename RAW, typename T, typename LOAD, typename FORM, typename OWN>
__device__ __forceinline__ void plane_rows(const CSRView<T>& A, const PlaneWalk& w, T* sm,
                                           LOAD load, FORM form, OWN own)
{
    constexpr int R = kWalkCols;
    constexpr uint32_t W = R * kBlock;
    const uint32_t S1 = A.udelta[5], span = W + 2 * S1, t = threadIdx.x;
    const int S2 = A.udelta[6], n = (int)A.nrow;
    for (uint32_t tile = blockIdx.x; tile < w.tiles; tile += gridDim.x) {
        const uint32_t seg = tile % w.segs, k0 = tile / w.segs * w.chunk;
        const uint32_t k1 = min(k0 + w.chunk, w.planes);
        const int c0 = (int)(seg * W);
        const int left = S2 + (int)S1 - c0; // columns from c0 on that any row here reads
        RAW cr[R], hr[2];
        bool cin[R], hin[2];
        // the operands of plane k: own columns, and (edges) the S1 columns on both sides
        auto fetch = [&](uint32_t k, bool edges) {
            const int base = (int)k * S2 + c0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int c = (int)t + r * kBlock;
                cin[r] = c < left && base + c < n;
                if (cin[r]) cr[r] = load((uint32_t)(base + c));
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t h = t + (uint32_t)i * kBlock;
                const int c = (int)(h < S1 ? h : h + W) - (int)S1;
                hin[i] = edges && h < 2 * S1 && c < left && base + c >= 0 && base + c < n;
                if (hin[i]) hr[i] = load((uint32_t)(base + c));
            }
        };
        // ... formed, shared (plane k's slot) and kept
        auto put = [&](uint32_t k, T (&v)[R]) {
            T* p = sm + (size_t)(k % 3) * span;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                v[r] = cin[r] ? form(cr[r]) : T(0);
                p[S1 + t + (uint32_t)r * kBlock] = v[r];
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t h = t + (uint32_t)i * kBlock;
                if (h < 2 * S1) p[h < S1 ? h : W + h] = hin[i] ? form(hr[i]) : T(0);
            }
        };
        auto masks = [&](uint32_t k, uint32_t (&m)[R]) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int c = c0 + (int)t + r * kBlock, row = (int)k * S2 + c;
                m[r] = c < S2 && row < n ? A.gnz ? grid_mask(A, (uint32_t)row)
                                                 : (uint32_t)__ldcs(A.mask + row)
                                         : 0u;
            }
        };
        T prev[R], cur[R], next[R];
        uint32_t m[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int c = (int)t + r * kBlock, row = ((int)k0 - 1) * S2 + c0 + c;
            prev[r] = row >= 0 && row < n && c < left ? form(load((uint32_t)row)) : T(0);
        }
        __syncthreads(); // the previous tile's slots are read
        masks(k0, m);
        fetch(k0, true);
        put(k0, cur);
        fetch(k0 + 1, k0 + 1 < k1);
        put(k0 + 1, next);
        __syncthreads();
        for (uint32_t k = k0; k < k1; ++k) {
            uint32_t mn[R];
            if (k + 1 < k1) {
                masks(k + 1, mn);
                fetch(k + 2, k + 2 < k1);
            }
            const T* p = sm + (size_t)(k % 3) * span + S1 + t;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int c = c0 + (int)t + r * kBlock, row = (int)k * S2 + c;
                if (c < S2 && row < n) {
                    const T* q = p + (uint32_t)r * kBlock;
                    const T a[7] = {prev[r], q[-(int)S1], q[-1], cur[r], q[1], q[S1], next[r]};
                    T s = T(0);
#pragma unroll
                    for (int u = 0; u < 7; ++u)
                        if ((m[r] >> u) & 1u) s = fma(A.uval[u], a[u], s);
                    own((size_t)row, cur[r], s);
                }
                prev[r] = cur[r];
                cur[r] = next[r];
            }
            if (k + 1 < k1) {
                put(k + 2, next); // the slot that plane k - 1 had
#pragma unroll
                for (int r = 0; r < R; ++r) m[r] = mn[r];
            }
            __syncthreads();
        }
    }
}

// Whether A can be walked: seven sorted offsets [-S2, -S1, -1, 0, 1, S1, S2] with
// 2 <= S1 <= kWalkS1 and S2 >= 2 S1, square.
template <typename T>
inline bool walkable(const CSRView<T>& A)
{
    const int32_t* d = A.udelta;
    return (A.mask || A.gnz) && A.ulen == 7 && A.nrow == A.mcol && A.nrow < 1u << 30 && d[3] == 0 &&
           d[2] == -1 && d[4] == 1 && d[1] == -d[5] && d[0] == -d[6] && d[5] >= 2 &&
           d[5] <= (int)kWalkS1 && d[6] >= 2 * d[5] && d[6] < 1 << 29;
}

// The walk of a walkable A for `resident` blocks, or none (tiles == 0) where an item would have
// fewer than kWalkChunk planes.
template <typename T>
inline PlaneWalk plane_walk(const CSRView<T>& A, int resident)
{
    constexpr uint32_t W = kWalkCols * kBlock;
    const uint32_t S2 = A.udelta[6];
    PlaneWalk w;
    w.planes = (A.nrow + S2 - 1) / S2;
    w.segs = (S2 + W - 1) / W;
    const uint32_t chunks = std::max(1u, std::min(w.planes, (uint32_t)resident / w.segs));
    w.chunk = (w.planes + chunks - 1) / chunks;
    if (w.chunk >= kWalkChunk) w.tiles = w.segs * ((w.planes + w.chunk - 1) / w.chunk);
    return w;
}

// The walk and the grid for kernel `kern` (no walk: grid 0).
struct WalkLaunch {
    PlaneWalk w;
    int grid = 0;
    size_t smem = 0;
};
template <typename T>
inline WalkLaunch walk_launch(const Ctx& c, const CSRView<T>& A, const void* kern)
{
    WalkLaunch l;
    if (!walkable(A)) return l;
    l.smem = walk_smem(A);
    const int g = resident_grid(c, kern, kBlock, l.smem);
    l.w = plane_walk(A, g);
    l.grid = std::min(g, (int)l.w.tiles);
    return l;
}

} // namespace fb
