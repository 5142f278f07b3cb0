// lu.cu -- partial-pivoting LU and the triangular solves built on it (FP64 plain form).
//
// Structure (a B200 re-design of InternalRecursiveMatrixLUDecompInPlace, LinAlgLU.pas:181-281):
//   * orders up to 512: the recursion splits the column range in two halves rounded to the
//     32-column leaf width (the reference halves exactly: mn div 2); larger orders: 256-column
//     outer panels with look-ahead, factored right-looking by leaves (lu_blocked below); the
//     leaves are factored by one thread-block cluster per panel with the panel resident in
//     distributed shared memory;
//   * a leaf's <= 32 row interchanges are applied at once to every other column of the matrix
//     (and to a row-permutation vector) by one swap launch, which replaces the reference's two
//     LUSwap calls per recursion level (:205, :237) -- the final matrix and pivot vector are the
//     same because each interchange is applied to every column exactly once, in order;
//   * A12 <- L11^{-1} A12 (LUBacksup :138-169) is a recursive triangular solve whose leaves run
//     a 32 x 32 register kernel and whose off-diagonal work goes through the DMMA GEMM;
//   * A22 -= A21 * A12 (MatrixMultEx ... doSub, :221) is the DMMA GEMM with the doSub epilogue.
// Pivot search follows the reference's leaf exactly: the largest |a| wins, the first (lowest
// row) among equals wins, a column whose largest |a| is <= 10/MaxDouble is singular (:246-268);
// the pivot column is scaled by the reciprocal 1/maxVal, as MatrixScaleAndAdd does.
#include <cooperative_groups.h>

#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"
#include "panel.cuh"

namespace cg = cooperative_groups;

namespace b2m {

constexpr int kPanelW = 32;  // largest leaf width

// ------------------------------------------------------------------------------------------
// Row interchanges of one leaf, applied to the columns [col_lo, col_hi) outside the leaf's own
// columns, to the permutation vector and (when given) to the outer panel's row map.  Warp 0 turns
// the <= 32 sequential swaps into a list of row moves.
// ------------------------------------------------------------------------------------------
constexpr int kSwapThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kSwapThreads)
    leaf_swap_kernel(T* A, int64_t ld, int col_lo, int col_hi, int c0, int w, const int32_t* ipiv, int32_t* perm,
                     int32_t* pmap, const int32_t* status) {
    __shared__ int src_main[kPanelW];
    __shared__ int mv_dst[2 * kPanelW], mv_src[2 * kPanelW];
    __shared__ int n_moves;
    if (status[kInfo] != 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < 32) {
        if (lane < w) src_main[lane] = c0 + lane;
        __syncwarp();
        int my_pos = -1, my_src = -1, n_extra = 0;
        const int qv = lane < w ? ipiv[c0 + lane] : 0;  // one load per lane, not w dependent loads
        for (int j = 0; j < w; ++j) {
            const int q = __shfl_sync(0xffffffffu, qv, j);
            if (q < c0 + w) {
                if (lane == 0 && q != c0 + j) {
                    const int t = src_main[j];
                    src_main[j] = src_main[q - c0];
                    src_main[q - c0] = t;
                }
            } else {
                const unsigned hit = __ballot_sync(0xffffffffu, my_pos == q);
                int owner;
                if (hit) {
                    owner = __ffs(hit) - 1;
                } else {
                    owner = n_extra++;
                    if (lane == owner) { my_pos = q; my_src = q; }
                }
                if (lane == owner) {
                    const int t = src_main[j];
                    src_main[j] = my_src;
                    my_src = t;
                }
            }
            __syncwarp();
        }
        // compact the moves (rows whose content changes)
        const bool mv_main = lane < w && src_main[lane] != c0 + lane;
        const bool mv_extra = lane < n_extra && my_src != my_pos;
        const unsigned bm = __ballot_sync(0xffffffffu, mv_main);
        const unsigned be = __ballot_sync(0xffffffffu, mv_extra);
        const int below = (1u << lane) - 1u;
        if (mv_main) {
            const int k = __popc(bm & below);
            mv_dst[k] = c0 + lane;
            mv_src[k] = src_main[lane];
        }
        if (mv_extra) {
            const int k = __popc(bm) + __popc(be & below);
            mv_dst[k] = my_pos;
            mv_src[k] = my_src;
        }
        if (lane == 0) n_moves = __popc(bm) + __popc(be);
    }
    __syncthreads();
    const int nm = n_moves;
    if (nm == 0) return;
    const int gc = col_lo + blockIdx.x * kSwapThreads + tid;
    const int col = gc < c0 ? gc : gc + w;  // the leaf's own columns are skipped
    if (col < col_hi) {
        T v[2 * kPanelW];
#pragma unroll
        for (int k = 0; k < 2 * kPanelW; ++k)
            if (k < nm) v[k] = A[(int64_t)mv_src[k] * ld + col];
#pragma unroll
        for (int k = 0; k < 2 * kPanelW; ++k)
            if (k < nm) A[(int64_t)mv_dst[k] * ld + col] = v[k];
    }
    if ((perm || pmap) && blockIdx.x == 0) {
        int pv = 0, qv = 0;
        if (tid < nm) {
            if (perm) pv = perm[mv_src[tid]];
            if (pmap) qv = pmap[mv_src[tid]];
        }
        __syncthreads();
        if (tid < nm) {
            if (perm) perm[mv_dst[tid]] = pv;
            if (pmap) pmap[mv_dst[tid]] = qv;
        }
    }
}

// Inside an outer panel of the blocked FP64 LU, right-looking by leaves: after a leaf is factored,
// (1) leaf_swap_u12_kernel applies its interchanges to the panel's other columns and, for the
// panel columns right of the leaf, turns the leaf's rows into U12 = L11^-1 A12 (thread per column:
// the <= 32 values of the column in the leaf's rows after the interchanges, then the unit-lower
// forward substitution with contributions in ascending order, as trsm_small_kernel computes it);
// (2) panel_rank_update_kernel subtracts L21 U12 from the rest of the panel (rows below the leaf).  Both
// only touch the outer panel's columns; the other columns get the panel's net permutation and one
// K = 256 update per panel.
constexpr int kSuThreads = 64;  // columns per CTA of leaf_swap_u12_kernel
template <typename T>
__global__ void __launch_bounds__(kSuThreads)
    leaf_swap_u12_kernel(T* A, int64_t ld, int col_lo, int col_hi, int c0, int w, const int32_t* ipiv, int32_t* perm,
                         int32_t* pmap, const int32_t* status) {
    __shared__ int src_main[kPanelW];
    __shared__ int mv_dst[2 * kPanelW], mv_src[2 * kPanelW];
    __shared__ int n_moves, n_main;
    __shared__ T s_l[kPanelW][kPanelW + 1];  // L11 (strictly lower part), s_l[j][i] = L(c0 + j, c0 + i)
    if (status[kInfo] != 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    batched_copy<kSuThreads, kPanelW * kPanelW / kSuThreads, T>(tid, kPanelW * kPanelW,
        [&](int e) {
            const int j = e / kPanelW, i = e - j * kPanelW;
            return (i < j && j < w) ? A[(int64_t)(c0 + j) * ld + c0 + i] : T(0);
        },
        [&](int e, T v) { s_l[e / kPanelW][e % kPanelW] = v; });
    if (tid < 32) {
        // The interchanges composed into moves.  Lane i holds sm = the original row whose content
        // ends in row c0 + i; lane e < n_extra holds a row q outside the leaf's rows that an
        // interchange reached (my_pos) and the original row whose content ends there (my_src).
        // Each interchange swaps two of these entries through shuffles (one warp, no shared
        // memory round trip per interchange).
        int sm = c0 + lane;
        int my_pos = -1, my_src = -1, n_extra = 0;
        const int qv = lane < w ? ipiv[c0 + lane] : 0;
        for (int j = 0; j < w; ++j) {
            const int q = __shfl_sync(0xffffffffu, qv, j);
            const int a = __shfl_sync(0xffffffffu, sm, j);
            if (q < c0 + w) {
                const int qi = q - c0;
                const int b = __shfl_sync(0xffffffffu, sm, qi);
                if (lane == j) sm = b;
                else if (lane == qi) sm = a;
            } else {
                const unsigned hit = __ballot_sync(0xffffffffu, my_pos == q);
                int owner;
                if (hit) {
                    owner = __ffs(hit) - 1;
                } else {
                    owner = n_extra++;
                    if (lane == owner) { my_pos = q; my_src = q; }
                }
                const int b = __shfl_sync(0xffffffffu, my_src, owner);
                if (lane == j) sm = b;
                if (lane == owner) my_src = a;
            }
        }
        if (lane < w) src_main[lane] = sm;
        const bool mv_main = lane < w && sm != c0 + lane;
        const bool mv_extra = lane < n_extra && my_src != my_pos;
        const unsigned bm = __ballot_sync(0xffffffffu, mv_main);
        const unsigned be = __ballot_sync(0xffffffffu, mv_extra);
        const int below = (1u << lane) - 1u;
        if (mv_main) {
            const int k = __popc(bm & below);
            mv_dst[k] = c0 + lane;
            mv_src[k] = sm;
        }
        if (mv_extra) {
            const int k = __popc(bm) + __popc(be & below);
            mv_dst[k] = my_pos;
            mv_src[k] = my_src;
        }
        if (lane == 0) { n_moves = __popc(bm) + __popc(be); n_main = __popc(bm); }
    }
    __syncthreads();
    const int nm = n_moves;
    const int gc = col_lo + blockIdx.x * kSuThreads + tid;
    const int col = (gc < c0 || col_lo >= c0 + w) ? gc : gc + w;  // the leaf's own columns are skipped
    if (col < col_hi) {
        // every read of this column happens before its first write
        if (col > c0) {  // right of the leaf: the leaf's rows after the interchanges, then U12
            // the moves into the leaf's rows are covered by x; only the moves out of them (the
            // extra entries, after the n_main moves into the leaf's rows) need their own values
            const int nmain = n_main, nx = nm - n_main;
            T x[kPanelW], v[kPanelW];
#pragma unroll
            for (int j = 0; j < kPanelW; ++j) x[j] = j < w ? A[(int64_t)src_main[j] * ld + col] : T(0);
#pragma unroll
            for (int e = 0; e < kPanelW; ++e)
                if (e < nx) v[e] = A[(int64_t)mv_src[nmain + e] * ld + col];
#pragma unroll
            for (int e = 0; e < kPanelW; ++e)
                if (e < nx) A[(int64_t)mv_dst[nmain + e] * ld + col] = v[e];
#pragma unroll
            for (int i = 0; i < kPanelW - 1; ++i) {
#pragma unroll
                for (int j = i + 1; j < kPanelW; ++j) x[j] = fma(-s_l[j][i], x[i], x[j]);
            }
#pragma unroll
            for (int j = 0; j < kPanelW; ++j)
                if (j < w) A[(int64_t)(c0 + j) * ld + col] = x[j];
        } else {
            T v[2 * kPanelW];
#pragma unroll
            for (int k = 0; k < 2 * kPanelW; ++k)
                if (k < nm) v[k] = A[(int64_t)mv_src[k] * ld + col];
#pragma unroll
            for (int k = 0; k < 2 * kPanelW; ++k)
                if (k < nm) A[(int64_t)mv_dst[k] * ld + col] = v[k];
        }
    }
    if ((perm || pmap) && blockIdx.x == 0 && nm > 0) {
        int pv = 0, qv = 0;
        if (tid < nm) {
            if (perm) pv = perm[mv_src[tid]];
            if (pmap) qv = pmap[mv_src[tid]];
        }
        __syncthreads();
        if (tid < nm) {
            if (perm) perm[mv_dst[tid]] = pv;
            if (pmap) pmap[mv_dst[tid]] = qv;
        }
    }
}

// A linked leaf [c0, c0 + w) (panel_kernel): its interchanges, given as moves, on the outer panel's
// columns left of it, [k0, c0), and on those beyond the next leaf, [nx, k1), where the leaf's rows
// also become U12 = L11^-1 A12.  32 columns per CTA of 4 warps; bound by latency (moves, rows, 32
// substitution steps), so all loads of a thread are in flight together and four lanes share a column
// of the substitution.  Runs on the leaf stream under the next leaf, whose time it must not exceed:
// leaf_swap_u12_kernel took 16 us for each side (it composes the interchanges itself, 3.7 us, and a
// thread owns a whole column), this takes 5.7 us for both.
constexpr int kLsThreads = 128;
__global__ void __launch_bounds__(kLsThreads) leaf_side_kernel(double* A, int64_t ld, int c0, int w, int k0, int nx,
                                                               int k1, const int32_t* moves, int32_t* perm,
                                                               int32_t* pmap, const int32_t* status) {
    __shared__ double s_x[kPanelW][kPanelW + 1], s_e[kPanelW][kPanelW + 1], s_l[kPanelW][kPanelW + 1];
    __shared__ int s_mv[3 * kPanelW + 1];
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const int nleft = (c0 - k0 + kPanelW - 1) / kPanelW;
    const bool right = (int)blockIdx.x >= nleft;
    const int cb = right ? nx + ((int)blockIdx.x - nleft) * kPanelW : k0 + (int)blockIdx.x * kPanelW;
    const int col = cb + lane, end = right ? k1 : c0;
    double l[kPanelW * kPanelW / kLsThreads];  // L11 (rows wp + 4 i, column `lane`)
#pragma unroll
    for (int i = 0; i < kPanelW / 4; ++i) {
        const int j = wp + 4 * i;
        l[i] = (right && j < w && lane < j) ? A[(int64_t)(c0 + j) * ld + c0 + lane] : 0.0;
    }
    if (t < 3 * kPanelW + 1) s_mv[t] = moves[t];
    __syncthreads();
    const int nx_rows = s_mv[kPanelW];
    double x[kPanelW / 4], e[kPanelW / 4];
#pragma unroll
    for (int i = 0; i < kPanelW / 4; ++i) {
        const int j = wp + 4 * i;
        x[i] = (col < end && j < w) ? A[(int64_t)s_mv[j] * ld + col] : 0.0;
        e[i] = (col < end && j < nx_rows) ? A[(int64_t)s_mv[2 * kPanelW + 1 + j] * ld + col] : 0.0;
    }
    int pv = 0, qv = 0, dst = -1;  // the maps: thread t < 32 the leaf's rows, t < 64 the others
    if (blockIdx.x == 0 && t < 2 * kPanelW) {
        const bool top = t < kPanelW;
        const int j = top ? t : t - kPanelW;
        if (top ? j < w : j < nx_rows) {
            const int src = s_mv[top ? j : 2 * kPanelW + 1 + j];
            dst = top ? c0 + j : s_mv[kPanelW + 1 + j];
            if (perm) pv = perm[src];
            if (pmap) qv = pmap[src];
        }
    }
#pragma unroll
    for (int i = 0; i < kPanelW / 4; ++i) {
        s_x[wp + 4 * i][lane] = x[i];
        s_e[wp + 4 * i][lane] = e[i];
        s_l[wp + 4 * i][lane] = l[i];
    }
    __syncthreads();  // every source of these columns, and of the maps, has been read
    if (dst >= 0) {
        if (perm) perm[dst] = pv;
        if (pmap) pmap[dst] = qv;
    }
    if (right) {
        // warp = 8 columns, lane = column + 8 * (row & 3); four rows a step, the finished element
        // broadcast by a shuffle; contributions in ascending order
        const int c = 8 * wp + (lane & 7), rg = lane >> 3;
#pragma unroll
        for (int i = 0; i < kPanelW / 4; ++i) x[i] = s_x[4 * i + rg][c];
#pragma unroll 1
        for (int q = 0; q < kPanelW / 4; ++q) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double xi = __shfl_sync(0xffffffffu, x[0], (lane & 7) + 8 * u);
                const double* lt = &s_l[4 * q + rg][4 * q + u];
                if (rg > u) x[0] = fma(-lt[0], xi, x[0]);
#pragma unroll
                for (int i = 1; i < kPanelW / 4; ++i)
                    if (q + i < kPanelW / 4) x[i] = fma(-lt[4 * i * (kPanelW + 1)], xi, x[i]);
            }
            s_x[4 * q + rg][c] = x[0];
#pragma unroll
            for (int i = 1; i < kPanelW / 4; ++i) x[i - 1] = x[i];
        }
        __syncthreads();
    }
    if (col < end) {
#pragma unroll
        for (int i = 0; i < kPanelW / 4; ++i) {
            const int j = wp + 4 * i;
            if (j < w && (right || s_mv[j] != c0 + j)) A[(int64_t)(c0 + j) * ld + col] = s_x[j][lane];
            if (j < nx_rows) A[(int64_t)s_mv[kPanelW + 1 + j] * ld + col] = s_e[j][lane];
        }
    }
}

// A[r][c] -= sum_{k < w} A[r][c0 + k] * A[c0 + k][c] for rows [r_lo, n) and columns [cl, ch): the
// leaf's rank-w update of the rest of its outer panel.  64 x 64 tiles, 4 x 4 per thread, the
// L21 and U12 slices staged in shared memory; the w products of each element are accumulated in
// ascending k and subtracted once (as the GEMM's doSub epilogue does).
// kSym (a Cholesky leaf): U12 is L21^T, and tiles strictly above the diagonal are left out.
constexpr int kRuT = 64;
template <bool kSym>
__global__ void __launch_bounds__(256, 2) panel_rank_update_kernel(double* A, int64_t ld, int n, int r_lo, int cl, int ch,
                                                          int c0, int w, const int32_t* status) {
    __shared__ double s_a[kRuT][kPanelW + 1];  // L21 rows of the tile
    __shared__ __align__(16) double s_b[kPanelW][kRuT];  // U12 columns of the tile
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int tiles_x = (ch - cl + kRuT - 1) / kRuT, tiles = tiles_x * ((n - r_lo + kRuT - 1) / kRuT);
    for (int tl = blockIdx.x; tl < tiles; tl += gridDim.x) {  // a grid smaller than the tiles loops
        const int r0 = r_lo + (tl / tiles_x) * kRuT, cb = cl + (tl % tiles_x) * kRuT;
        if (kSym && r0 + kRuT <= cb) continue;
        batched_copy<256, kRuT * kPanelW / 256, double>(t, kRuT * kPanelW,
            [&](int e) {
                const int rr = e >> 5, k = e & 31, row = r0 + rr;
                return (row < n && k < w) ? A[(int64_t)row * ld + c0 + k] : 0.0;
            },
            [&](int e, double v) { s_a[e >> 5][e & 31] = v; });
        batched_copy<256, kPanelW * kRuT / 256, double>(t, kPanelW * kRuT,
            [&](int e) {
                const int k = kSym ? e & 31 : e / kRuT, col = cb + (kSym ? e >> 5 : e % kRuT);
                if (k >= w || col >= ch) return 0.0;
                return kSym ? A[(int64_t)col * ld + c0 + k] : A[(int64_t)(c0 + k) * ld + col];
            },
            [&](int e, double v) { s_b[kSym ? e & 31 : e / kRuT][kSym ? e >> 5 : e % kRuT] = v; });
        // the tile's own values, loaded while the slices arrive
        double c[4][4];
    #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + 4 * ty + i;
    #pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int col = cb + 4 * tx + j;
                c[i][j] = (row < n && col < ch) ? A[(int64_t)row * ld + col] : 0.0;
            }
        }
        __syncthreads();
        double acc[4][4];
    #pragma unroll
        for (int i = 0; i < 4; ++i)
    #pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    #pragma unroll 8
        for (int k = 0; k < kPanelW; ++k) {
            const double2 b01 = *reinterpret_cast<const double2*>(&s_b[k][4 * tx]);
            const double2 b23 = *reinterpret_cast<const double2*>(&s_b[k][4 * tx + 2]);
            const double bv[4] = {b01.x, b01.y, b23.x, b23.y};
    #pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double av = s_a[4 * ty + i][k];
    #pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(av, bv[j], acc[i][j]);
            }
        }
    #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + 4 * ty + i;
    #pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int col = cb + 4 * tx + j;
                if (row < n && col < ch) A[(int64_t)row * ld + col] = c[i][j] - acc[i][j];
            }
        }
        __syncthreads();  // the tile's slices are no longer read
    }
}

// U12 = L11^-1 A12 for one outer panel in a single launch, and the diagonal blocks of the solves with many right-hand
// sides: L11 unit lower or, kUpper, upper (k <= 256 rows, at L with row stride ldl, from the last block up), the
// right-hand sides k x ncols at B.  A CTA owns NC columns, held in shared memory
// for the whole solve; per 32-row block of L11 (its block column staged by cp.async, the next one
// while the current one is used) one warp per 8 columns substitutes the block's triangle, four lanes
// a column (contributions in ascending order), and all warps subtract the block's contribution from
// the rows below it on the FP64 tensor cores.  What bounds it is the chain of the eight blocks, so
// the columns of the next panel, which are on the critical path, run eight to a CTA (32 CTAs for 256
// columns), and only right-hand sides beyond what one wave holds so run 32 to a CTA, which reads L11
// a quarter as often.  256 rows, 256 columns: 60 us before (32 columns a CTA, one warp substituting a
// 32 x 32 triangle from unrolled code), 25.6 us with 8 columns a CTA, 39 us with 32.
constexpr int kTpK = 256;   // rows of the panel
constexpr int kTpThreads = 256;
constexpr int kTpPitch = kTpK + 4;  // columns of X in shared memory (column-major; conflict-free fragments)
template <int NC> constexpr int tp_smem() { return (NC * kTpPitch + 2 * kTpK * kPanelW) * (int)sizeof(double); }

// Back substitution with a block's upper triangle (identity past its rows): lane = column + 8 * (row & 3), x its
// rows 4 e + (lane >> 3); results to xc.  x / d is the product with the reciprocal corrected by its exact residual
// (as accurate as the division, whose 144 cycles would be on the chain 32 times); with divisions where a
// diagonal is far from 1, and in the columns with a result that is not finite.  So a column's result does not
// depend on its neighbours.
__device__ __forceinline__ void tp_upper(const double (*s_t)[kPanelW + 1], int lane, const double (&y)[kPanelW / 4],
                                         double* xc) {
    constexpr int kTop = kPanelW / 4 - 1;
    const int rg = lane >> 3;
    double dv[kTop + 1], di[kTop + 1];
    bool odd = false;
#pragma unroll
    for (int e = 0; e <= kTop; ++e) {
        dv[e] = s_t[4 * e + rg][4 * e + rg];
        di[e] = 1.0 / dv[e];
        odd = odd || mag_hi(dv[e]) - 0x01700000u >= 0x7d000000u;  // outside 2^-1000 .. 2^1000
    }
    auto solve = [&](auto divide, bool put) {
        double x[kTop + 1], d[kTop + 1], r[kTop + 1];
#pragma unroll
        for (int e = 0; e <= kTop; ++e) {
            x[e] = y[e];
            d[e] = dv[e];
            r[e] = di[e];
        }
        bool finite = true;
#pragma unroll 1
        for (int q = kTop; q >= 0; --q) {
#pragma unroll
            for (int u = 3; u >= 0; --u) {
                const double z = x[kTop];
                double xq;
                if constexpr (decltype(divide)::value) {
                    xq = z / d[kTop];
                } else {
                    xq = z * r[kTop];
                    xq = fma(fma(-xq, d[kTop], z), r[kTop], xq);
                }
                const double xj = __shfl_sync(0xffffffffu, xq, (lane & 7) + 8 * u);
                if (rg == u) x[kTop] = xq;
                const double* uc = &s_t[rg][4 * q + u];
                if (rg < u) x[kTop] = fma(-uc[4 * q * (kPanelW + 1)], xj, x[kTop]);
#pragma unroll
                for (int e = 1; e <= kTop; ++e)
                    if (q - e >= 0) x[kTop - e] = fma(-uc[4 * (q - e) * (kPanelW + 1)], xj, x[kTop - e]);
            }
            finite = finite && mag_hi(x[kTop]) < kInfHi;
            if (put) xc[4 * q + rg] = x[kTop];
#pragma unroll
            for (int e = kTop; e > 0; --e) {
                x[e] = x[e - 1];
                d[e] = d[e - 1];
                r[e] = r[e - 1];
            }
        }
        return finite;
    };
    uint32_t again = __any_sync(0xffffffffu, odd) ? 0xffffffffu : 0u;
    if (!again) again = __ballot_sync(0xffffffffu, !solve(std::false_type{}, true));
    if (again) solve(std::true_type{}, (again & (0x01010101u << (lane & 7))) != 0);
}

template <int NC, bool kUpper>
__global__ void __launch_bounds__(kTpThreads, 1) trsm_panel_kernel(const double* L, int64_t ldl, double* B,
                                                                   int64_t ldb, int k, int ncols,
                                                                   const int32_t* status) {
    extern __shared__ __align__(16) double tp_dyn[];
    double* s_l = tp_dyn;                         // [2][kTpK][kPanelW] block columns of L11, pairs swizzled by row
    double* s_x = tp_dyn + 2 * kTpK * kPanelW;    // [NC][kTpPitch] this CTA's columns (zero past row k)
    __shared__ double s_t[kPanelW][kPanelW + 1];  // the block's triangle
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int cb = blockIdx.x * NC;
    const int nb = (int)ceil_div(k, kPanelW);
    auto sx = [](int row, int c) { return row * kPanelW + 2 * ((c >> 1) ^ (row & 7)) + (c & 1); };
    // block column i of the triangle: columns [32 i, 32 i + 32), rows from 32 i on (kUpper: rows up to and with
    // the block's) -> buffer `buf` (16-byte pieces)
    auto stage = [&](int i, int buf) {
        double* dst = s_l + buf * kTpK * kPanelW;
        const int r0 = kPanelW * i, c = 2 * (t & 15), col = r0 + c, first = kUpper ? 0 : r0;
        const int rows = kUpper ? min(k, r0 + kPanelW) : k - r0;
        const int bytes = col + 1 < k ? 16 : (col < k ? 8 : 0);
        const double* src = L + (int64_t)first * ldl + (col < k ? col : 0);
#pragma unroll 4
        for (int r = t >> 4; r < rows; r += kTpThreads / 16) cp_async16(dst + sx(r, c), src + (int64_t)r * ldl, bytes);
        cp_async_commit();
    };
    stage(kUpper ? nb - 1 : 0, 0);
    batched_copy<kTpThreads, 8, double>(t, kTpK * NC,
        [&](int e) {
            const int r = e / NC, c = e % NC;
            return (r < k && cb + c < ncols) ? B[(int64_t)r * ldb + cb + c] : 0.0;
        },
        [&](int e, double v) { s_x[(e % NC) * kTpPitch + e / NC] = v; });
    for (int step = 0; step < nb; ++step) {
        const int i = kUpper ? nb - 1 - step : step;
        if (step + 1 < nb) {
            stage(kUpper ? i - 1 : i + 1, (step + 1) & 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const double* lb = s_l + (step & 1) * kTpK * kPanelW;  // lb[sx(r - 32 i, q)] = L[r][32 i + q]; kUpper: lb[sx(r, q)]
        const int r0 = kPanelW * i, bw = min(kPanelW, k - r0);
        for (int e = t; e < kPanelW * kPanelW; e += kTpThreads) {  // the triangle, for constant offsets below
            const int r = e >> 5, c = e & 31;
            if constexpr (kUpper) s_t[r][c] = (c < bw && r <= c) ? lb[sx(r0 + r, c)] : (r == c ? 1.0 : 0.0);
            else s_t[r][c] = (r < bw && c < r) ? lb[sx(r, c)] : 0.0;
        }
        __syncthreads();
        if (warp < NC / 8) {
            // warp = 8 columns, lane = column + 8 * (row & 3); rows past the end are zero and stay so
            double* xc = s_x + (8 * warp + (lane & 7)) * kTpPitch + r0;
            const int rg = lane >> 3;
            double x[kPanelW / 4];
#pragma unroll
            for (int e = 0; e < kPanelW / 4; ++e) x[e] = xc[4 * e + rg];
            if constexpr (kUpper) tp_upper(s_t, lane, x, xc);
            const double* lt = &s_t[rg][0];
#pragma unroll 1
            for (int q = 0; !kUpper && q < kPanelW / 4; ++q, lt += 4 * (kPanelW + 1) + 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const double xi = __shfl_sync(0xffffffffu, x[0], (lane & 7) + 8 * u);
                    if (rg > u) x[0] = fma(-lt[u], xi, x[0]);
#pragma unroll
                    for (int e = 1; e < kPanelW / 4; ++e)
                        if (q + e < kPanelW / 4) x[e] = fma(-lt[4 * e * (kPanelW + 1) + u], xi, x[e]);
                }
                xc[4 * q + rg] = x[0];
#pragma unroll
                for (int e = 1; e < kPanelW / 4; ++e) x[e - 1] = x[e];
            }
        }
        __syncthreads();
        // rows below the block (only full blocks have any; kUpper: above it), 16 x 8 tiles:
        // a = L[g][k + tq], L[g + 8][k + tq], b = x[k + tq][g], c = rows g, g + 8, columns 2 tq, 2 tq + 1
        const int g = lane >> 2, tq = lane & 3;
        const int mt = (kUpper ? r0 : k - r0 - bw + 15) / 16, row0 = kUpper ? 0 : r0;
        for (int tile = warp; tile < mt * (NC / 8); tile += kTpThreads / 32) {
            const int c8 = 8 * (tile % (NC / 8)), ra = (kUpper ? 0 : bw) + 16 * (tile / (NC / 8)) + g, rb = ra + 8;
            const bool oka = row0 + ra < k, okb = row0 + rb < k;
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            const double* xb = s_x + (c8 + g) * kTpPitch + r0 + tq;
#pragma unroll
            for (int q = 0; q < kPanelW / 4; ++q) {
                const double a0 = oka ? lb[sx(ra, 4 * q + tq)] : 0.0, a1 = okb ? lb[sx(rb, 4 * q + tq)] : 0.0;
                const double b0 = xb[4 * q];
                asm volatile(
                    "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                    : "+d"(acc[0]), "+d"(acc[1]), "+d"(acc[2]), "+d"(acc[3])
                    : "d"(a0), "d"(a1), "d"(b0));
            }
            double* xd = s_x + (c8 + 2 * tq) * kTpPitch + row0;
            if (oka) { xd[ra] -= acc[0]; xd[kTpPitch + ra] -= acc[1]; }
            if (okb) { xd[rb] -= acc[2]; xd[kTpPitch + rb] -= acc[3]; }
        }
        __syncthreads();  // the buffer of this step is restaged for the one after the next
    }
    for (int e = t; e < kTpK * NC; e += kTpThreads) {
        const int r = e / NC, c = e % NC;
        if (r < k && cb + c < ncols) B[(int64_t)r * ldb + cb + c] = s_x[c * kTpPitch + r];
    }
}

// The outer panel's net row permutation applied to the columns [col_begin, col_end) outside it:
// row i of the rows [oc0, n) receives what row pmap[i] held when the panel started.  CTA per 32
// columns; each CTA lists the moved rows (at most 2 x 256 for a 256-column panel; warp-aggregated
// appends) and loads all of their sources into registers before any write.
constexpr int kPpMax = 512;
__global__ void __launch_bounds__(256) panel_permute_f64_kernel(double* A, int64_t ld, int n, int oc0, int col_begin,
                                                                int col_end, const int32_t* pmap, int32_t* status) {
    __shared__ int s_dst[kPpMax], s_src[kPpMax], s_cnt;
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31;
    if (t == 0) s_cnt = 0;
    __syncthreads();
    constexpr int kScan = 16;  // row-map entries per thread per pass, all loaded before use
    for (int p0 = oc0; p0 < n; p0 += 256 * kScan) {
        int src[kScan];
#pragma unroll
        for (int u = 0; u < kScan; ++u) {
            const int i = p0 + 256 * u + t;
            src[u] = i < n ? pmap[i] : i;
        }
#pragma unroll
        for (int u = 0; u < kScan; ++u) {
            const int i = p0 + 256 * u + t;
            const bool mv = src[u] != i;
            const unsigned bal = __ballot_sync(0xffffffffu, mv);
            if (!bal) continue;  // warp-uniform
            int base = 0;
            if (lane == 0) base = atomicAdd(&s_cnt, __popc(bal));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (mv) {
                const int k = base + __popc(bal & ((1u << lane) - 1u));
                if (k < kPpMax) { s_dst[k] = i; s_src[k] = src[u]; }
            }
        }
    }
    __syncthreads();
    const int cnt = s_cnt;
    if (cnt > kPpMax) {  // a 256-column panel moves at most 512 rows; anything else is an internal error
        if (t == 0) atomicExch(&status[kTimeout], 202);
        return;
    }
    const int col = col_begin + blockIdx.x * 32 + lane, rg = t >> 5;
    const bool ok = col < col_end;
    double x[kPpMax / 8];
#pragma unroll
    for (int q = 0; q < kPpMax / 8; ++q) {
        const int k = rg + 8 * q;
        x[q] = (ok && k < cnt) ? A[(int64_t)s_src[k] * ld + col] : 0.0;
    }
    __syncthreads();  // every source of this CTA's columns is read before any row is written
#pragma unroll
    for (int q = 0; q < kPpMax / 8; ++q) {
        const int k = rg + 8 * q;
        if (ok && k < cnt) A[(int64_t)s_dst[k] * ld + col] = x[q];
    }
}

// ------------------------------------------------------------------------------------------
// Small triangular solves (k <= 32) on a strip of columns.  One warp handles 4 columns; lane i
// holds row i of the triangle (registers) and x_i of each column; at step j the final x_j is
// broadcast with a shuffle and every later row subtracts its multiple, so the dependent chain is
// 32 shuffle+FMA steps.  Lower: unit diagonal, contributions in ascending j (LUBacksup and the
// forward sweep of MatrixLUBackSubst).  Upper: x_j = (b_j - sum) / U[j][j] with a true division
// (the backward sweep, LinAlgLU.pas:362-382), contributions in descending j.
// ------------------------------------------------------------------------------------------
constexpr int kTrsmThreads = 128;
constexpr int kTrsmCpw = 4;  // columns per warp

template <typename T>
__global__ void __launch_bounds__(kTrsmThreads)
    trsm_small_kernel(const T* L, int64_t ldl, T* B, int64_t ldb, int k, int ncols, int upper,
                      const int32_t* status) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = (blockIdx.x * (kTrsmThreads / 32) + warp) * kTrsmCpw;
    // all global loads first: the status word, this lane's row of the triangle, its x values
    const int32_t st = status ? status[kInfo] : 0;
    T lrow[kPanelW];
#pragma unroll
    for (int j = 0; j < kPanelW; ++j) lrow[j] = (lane < k && j < k) ? L[(int64_t)lane * ldl + j] : T(0);
    T x[kTrsmCpw];
#pragma unroll
    for (int q = 0; q < kTrsmCpw; ++q)
        x[q] = (lane < k && c0 + q < ncols) ? B[(int64_t)lane * ldb + c0 + q] : T(0);
    if (st != 0 || c0 >= ncols) return;
    if (!upper) {
#pragma unroll
        for (int j = 0; j < kPanelW - 1; ++j) {
            if (j >= k) break;
#pragma unroll
            for (int q = 0; q < kTrsmCpw; ++q) {
                const T xj = __shfl_sync(0xffffffffu, x[q], j);
                if (lane > j) x[q] = fma(-lrow[j], xj, x[q]);
            }
        }
    } else {
#pragma unroll
        for (int j = kPanelW - 1; j >= 0; --j) {
            if (j >= k) continue;
#pragma unroll
            for (int q = 0; q < kTrsmCpw; ++q) {
                if (lane == j) x[q] = x[q] / lrow[j];
                const T xj = __shfl_sync(0xffffffffu, x[q], j);
                if (lane < j) x[q] = fma(-lrow[j], xj, x[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kTrsmCpw; ++q)
        if (lane < k && c0 + q < ncols) B[(int64_t)lane * ldb + c0 + q] = x[q];
}

__global__ void iota_kernel(int32_t* v, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (int32_t)i;
}

// X[i][:] = B[perm[i]][:]
__global__ void gather_rows_kernel(double* X, int64_t ldx, const double* B, int64_t ldb, const int32_t* perm,
                                   int64_t n, int64_t nrhs) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * nrhs) return;
    const int64_t i = e / nrhs, c = e - i * nrhs;
    X[i * ldx + c] = B[(int64_t)perm[i] * ldb + c];
}

// perm from a LAPACK-style ipiv: the result of the sequential interchanges of 0, 1, 2, ...
//
// Where every interchange reaches forward (i <= ipiv[i] < n or out of range, which means none), the
// content a position has at a step follows from the last earlier interchange that reached it: with
// V(j) the content of position j before step j,
//     V(j) = V(k), k the last k < j with ipiv[k] = j, or j if there is none;
//     perm[i] = V(i) if ipiv[i] = i, else V(k), k the last k < i with ipiv[k] = ipiv[i], or ipiv[i].
// The first k is a maximum over all interchanges; the second comes from one warp walking the steps 32
// at a time with a table of the last interchange per position; V by pointer jumping.  Order 4096 takes
// 37 us; one thread's sequential interchanges (140 cycles each), which remain for other vectors and
// orders, take 283.
constexpr int kPermThreads = 1024;
constexpr uint16_t kPermNone = 0xffff;
constexpr int kPermMax = 32768;  // orders whose three tables of 16-bit indices fit shared memory
__global__ void __launch_bounds__(kPermThreads) perm_from_ipiv_kernel(const int32_t* ipiv, int n, int32_t* perm) {
    extern __shared__ __align__(16) uint16_t pi_dyn[];
    uint16_t* up = pi_dyn;            // the targets; then V's pointers: up[j] = the k of V(j), or j
    uint16_t* last = pi_dyn + n;      // position -> last interchange that reached it so far
    uint16_t* prev = pi_dyn + 2 * n;  // i -> the last k < i with ipiv[k] = ipiv[i]
    __shared__ int s_back;
    const int t = threadIdx.x, lane = t & 31;
    auto target = [&](int i) {
        const int q = ipiv[i];
        return q >= 0 && q < n ? q : i;
    };
    if (t == 0) s_back = 0;
    __syncthreads();
    for (int i = t; i < n; i += kPermThreads) {
        const int q = target(i);
        up[i] = (uint16_t)q;
        last[i] = kPermNone;
        if (q < i) s_back = 1;
    }
    __syncthreads();
    if (s_back) {  // an interchange that reaches back: step by step, `last` as the permutation
        for (int i = t; i < n; i += kPermThreads) last[i] = (uint16_t)i;
        __syncthreads();
        if (t == 0)
            for (int i = 0; i < n; ++i) {
                const int q = up[i];
                const uint16_t v = last[i];
                last[i] = last[q];
                last[q] = v;
            }
        __syncthreads();
        for (int i = t; i < n; i += kPermThreads) perm[i] = last[i];
        return;
    }
    if (t < 32) {
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane, q = i < n ? up[i] : -1 - lane;
            const uint32_t same = __match_any_sync(0xffffffffu, q);
            const uint32_t before = same & ((1u << lane) - 1u);
            if (i < n) prev[i] = before ? (uint16_t)(i0 + 31 - __clz(before)) : last[q];
            __syncwarp();
            if (i < n && (same >> lane) == 1u) last[q] = (uint16_t)i;  // the chunk's last one
            __syncwarp();
        }
    }
    __syncthreads();
    // `last` now holds, per position, its last interchange of all: of its own step (none before) or
    // the last earlier one; a position's own step that moves nothing hides the earlier one
    for (int j = t; j < n; j += kPermThreads) {
        uint16_t k = last[j];
        if (k == (uint16_t)j) k = prev[j];
        up[j] = k != kPermNone ? k : (uint16_t)j;
    }
    __syncthreads();
    // up[j] -> the root of j's chain: every value ever read is one of j's ancestors, so the threads need
    // not agree on a round's old and new values, and a round in which nothing moved ends it
    volatile uint16_t* vup = up;
    for (;;) {
        int moved = 0;
        for (int j = t; j < n; j += kPermThreads) {
            const uint16_t u = vup[j], v = vup[u];
            if (v != u) {
                vup[j] = v;
                moved = 1;
            }
        }
        if (!__syncthreads_or(moved)) break;
    }
    for (int i = t; i < n; i += kPermThreads) {
        const int q = target(i);
        perm[i] = q == i ? up[i] : (prev[i] != kPermNone ? up[prev[i]] : q);
    }
}

// the same for larger orders, step by step: on a copy in shared memory while n ints fit there, else in global memory
__global__ void perm_from_ipiv_serial_kernel(const int32_t* ipiv, int n, int32_t* perm, int in_smem) {
    extern __shared__ int32_t ps_dyn[];
    int32_t* pv = in_smem ? ps_dyn : perm;
    for (int i = threadIdx.x; i < n; i += blockDim.x) pv[i] = i;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < n; ++i) {
            const int q = ipiv[i];
            if (q != i && q >= 0 && q < n) {
                const int t = pv[i];
                pv[i] = pv[q];
                pv[q] = t;
            }
        }
    }
    __syncthreads();
    if (in_smem)
        for (int i = threadIdx.x; i < n; i += blockDim.x) perm[i] = pv[i];
}

// det = (-1)^{#i: ipiv[i] != i} * U[0][0] * U[1][1] * ... in this order (MatrixDeterminant :467-476);
// the diagonal is staged through shared memory 1024 entries at a time (launch with 1024 threads)
constexpr int kDetChunk = 1024;
__global__ void __launch_bounds__(kDetChunk)
    determinant_kernel(const double* LU, int64_t ld, int n, const int32_t* ipiv, const int32_t* status, double* det) {
    __shared__ double dg[kDetChunk];
    __shared__ int flips;
    if (threadIdx.x == 0) flips = 0;
    __syncthreads();
    int local = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (ipiv[i] != i) local++;
    atomicAdd(&flips, local);
    __syncthreads();
    double r = (flips & 1) ? -1.0 : 1.0;  // thread 0's running product
    for (int c0 = 0; c0 < n; c0 += kDetChunk) {
        const int i = c0 + (int)threadIdx.x;
        if (i < n) dg[threadIdx.x] = LU[(int64_t)i * ld + i];
        __syncthreads();
        if (threadIdx.x == 0) {
            const int cnt = min(kDetChunk, n - c0);
            for (int k = 0; k < cnt; ++k) r = r * dg[k];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *det = status[kInfo] != 0 ? 0.0 : r;
}

// ------------------------------------------------------------------------------------------
// host drivers
// ------------------------------------------------------------------------------------------
namespace {

int64_t split_cols(int64_t w) { return round_up((w + 1) / 2, kPanelW); }

void CUDART_CB progress_trampoline(void* p) {
    const ProgressNote* note = static_cast<const ProgressNote*>(p);
    if (note->fn) note->fn(note->percent, note->user);
}

// TLinEquProgress, queued behind the work on `st`: columns factored * 100 div n
int32_t report_progress(Ctx* ctx, cudaStream_t st, int64_t columns, int64_t n) {
    if (!ctx->progress || ctx->progress_notes.size() >= ctx->progress_notes.capacity()) return B2M_OK;
    ctx->progress_notes.push_back(ProgressNote{ctx->progress, ctx->progress_user, (int32_t)(columns * 100 / n)});
    B2M_CU(ctx, cudaLaunchHostFunc(st, progress_trampoline, &ctx->progress_notes.back()));
    return B2M_OK;
}

// the leaf's interchanges on columns [col_lo, col_hi) (which contain the leaf's own columns)
template <typename T>
int32_t launch_swaps_range(Ctx* ctx, cudaStream_t st, T* A, int64_t ld, int col_lo, int col_hi, int c0, int w,
                           const int32_t* ipiv, int32_t* perm, int32_t* pmap) {
    const int other = col_hi - col_lo - w;
    const int blocks = std::max(1, (int)ceil_div(other, kSwapThreads));
    prof_begin(ctx, st, kClsSwap);
    leaf_swap_kernel<T><<<blocks, kSwapThreads, 0, st>>>(A, ld, col_lo, col_hi, c0, w, ipiv, perm, pmap,
                                                         ctx->d_status);
    prof_end(ctx, st, kClsSwap, 4.0 * w * other * sizeof(T));  // <= 2w rows read + written
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

template <typename T>
int32_t launch_swaps_impl(Ctx* ctx, cudaStream_t st, T* A, int64_t ld, int ncols, int c0, int w, const int32_t* ipiv,
                     int32_t* perm) {
    return launch_swaps_range<T>(ctx, st, A, ld, 0, ncols, c0, w, ipiv, perm, nullptr);
}

template <typename T>
int32_t launch_trsm_small_impl(Ctx* ctx, cudaStream_t st, const T* L, int64_t ldl, T* B, int64_t ldb, int k, int ncols,
                          bool upper) {
    if (k <= 0 || ncols <= 0) return B2M_OK;
    const int blocks = (int)ceil_div(ncols, (kTrsmThreads / 32) * kTrsmCpw);
    prof_begin(ctx, st, kClsTrsm);
    trsm_small_kernel<T><<<blocks, kTrsmThreads, 0, st>>>(L, ldl, B, ldb, k, ncols, upper ? 1 : 0, ctx->d_status);
    prof_end(ctx, st, kClsTrsm, (double)sizeof(T) * (k * k + 2.0 * k * ncols));  // bytes
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

// Triangular operand description for the recursive solves: the triangle T lives in the
// row-major array (Abase, lda, an n x n extent) at diagonal offset r0; the right-hand sides are
// rows [br0, br0+k) and columns [bc0, bc0+ncols) of (Bbase, ldb) whose map extent is bn x bcols.
struct TriSolve {
    const double* A;
    int64_t lda, n;
    double* B;
    int64_t ldb, bn, bcols, bc0, ncols;
};

// B (k <= 256 rows, ncols columns) <- T^-1 B in one launch, T unit lower or upper.  8 columns a CTA while
// the SMs hold them all, then 32.
int32_t launch_trsm_panel(Ctx* ctx, cudaStream_t st, const double* T, int64_t ldt, double* B, int64_t ldb, int k,
                          int64_t ncols, bool upper) {
    const bool few = ncols <= 8 * ctx->num_sms;
    const auto kern = upper ? (few ? trsm_panel_kernel<8, true> : trsm_panel_kernel<32, true>)
                            : (few ? trsm_panel_kernel<8, false> : trsm_panel_kernel<32, false>);
    const int smem = few ? tp_smem<8>() : tp_smem<32>();
    std::atomic<int>& attr = device_flag((const void*)kern, 0, ctx->device);
    if (!attr.load()) {
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr.store(1);
    }
    prof_begin(ctx, st, kClsTrsm);
    B2M_CU(ctx, launch_k(ctx, kern, dim3((unsigned)ceil_div(ncols, few ? 8 : 32)), dim3(kTpThreads), (size_t)smem, st,
                         T, ldt, B, ldb, k, (int)ncols, (const int32_t*)ctx->d_status));
    prof_end(ctx, st, kClsTrsm, 8.0 * (k * (double)k / 2 + 2.0 * k * (double)ncols));  // bytes
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

// Whether a diagonal block of the recursive solves goes to launch_trsm_panel (which wants 16-byte aligned pairs of
// the triangle), and where a larger one is split.  Down to 32 rows by recursion, with a
// product at every level, the inverse of order 512 took 977 us, of order 1500 3.56 ms; with blocks of 256 rows in one
// launch 680 us and 2.70 ms.
bool trsm_whole(const TriSolve& t, int64_t k) { return k <= kTpK && (t.lda & 1) == 0 && aligned16(t.A); }
int64_t trsm_split(int64_t k) { return k > kTpK ? round_up((k + 1) / 2, kTpK) : split_cols(k); }

int32_t trsm_lower_rec(Ctx* ctx, cudaStream_t st, const TriSolve& t, int64_t r0, int64_t br0, int64_t k) {
    if (k <= kPanelW)
        return launch_trsm_small_impl<double>(ctx, st, t.A + r0 * t.lda + r0, t.lda, t.B + br0 * t.ldb + t.bc0, t.ldb,
                                         (int)k, (int)t.ncols, false);
    if (trsm_whole(t, k))
        return launch_trsm_panel(ctx, st, t.A + r0 * t.lda + r0, t.lda, t.B + br0 * t.ldb + t.bc0, t.ldb, (int)k,
                                 t.ncols, false);
    const int64_t k1 = trsm_split(k), k2 = k - k1;
    B2M_TRY(trsm_lower_rec(ctx, st, t, r0, br0, k1));
    DOperand a{t.A, t.lda, t.n, t.n, r0 + k1, r0, true};
    DOperand b{t.B, t.ldb, t.bn, t.bcols, br0, t.bc0, false};
    B2M_TRY(dgemm_tiled(ctx, st, a, b, t.B + (br0 + k1) * t.ldb + t.bc0, t.ldb, k2, t.ncols, k1, B2M_DO_SUB, true));
    return trsm_lower_rec(ctx, st, t, r0 + k1, br0 + k1, k2);
}

int32_t trsm_upper_rec(Ctx* ctx, cudaStream_t st, const TriSolve& t, int64_t r0, int64_t br0, int64_t k) {
    if (k <= kPanelW)
        return launch_trsm_small_impl<double>(ctx, st, t.A + r0 * t.lda + r0, t.lda, t.B + br0 * t.ldb + t.bc0, t.ldb,
                                         (int)k, (int)t.ncols, true);
    if (trsm_whole(t, k))
        return launch_trsm_panel(ctx, st, t.A + r0 * t.lda + r0, t.lda, t.B + br0 * t.ldb + t.bc0, t.ldb, (int)k,
                                 t.ncols, true);
    const int64_t k1 = trsm_split(k), k2 = k - k1;
    B2M_TRY(trsm_upper_rec(ctx, st, t, r0 + k1, br0 + k1, k2));
    DOperand a{t.A, t.lda, t.n, t.n, r0, r0 + k1, true};
    DOperand b{t.B, t.ldb, t.bn, t.bcols, br0 + k1, t.bc0, false};
    B2M_TRY(dgemm_tiled(ctx, st, a, b, t.B + br0 * t.ldb + t.bc0, t.ldb, k1, t.ncols, k2, B2M_DO_SUB, true));
    return trsm_upper_rec(ctx, st, t, r0, br0, k1);
}

// where a leaf's interchanges go: the columns [col_lo, col_hi) (the whole matrix, or one outer
// panel whose other columns are permuted once per panel through the row map pmap)
struct SwapScope {
    int64_t col_lo, col_hi;
    int32_t* pmap;
};

// factor columns [c0, c0+width), rows [c0, n); leaves of at most `leaf` columns
int32_t lu_rec(Ctx* ctx, cudaStream_t st, double* A, int64_t ld, int64_t n, int64_t c0, int64_t width,
               int32_t* ipiv, int32_t* perm, int64_t leaf, const SwapScope& sc) {
    if (width <= leaf) {
        B2M_TRY(launch_panel<double>(ctx, st, A + c0 * ld + c0, ld, (int)(n - c0), (int)width, (int)c0, (int)c0,
                                     ipiv));
        B2M_TRY(launch_swaps_range<double>(ctx, st, A, ld, (int)sc.col_lo, (int)sc.col_hi, (int)c0, (int)width, ipiv,
                                           perm, sc.pmap));
        return B2M_OK;
    }
    // splits on multiples of 16 above the leaf level keep the Schur GEMMs' K on whole TMA k-tiles
    // (8-column leaves then meet only in their own narrow K = 8 updates)
    const int64_t step = width > 16 ? std::max<int64_t>(leaf, 16) : leaf;
    const int64_t nleft = round_up((width + 1) / 2, step), nright = width - nleft;
    B2M_TRY(lu_rec(ctx, st, A, ld, n, c0, nleft, ipiv, perm, leaf, sc));
    // A12 <- L11^{-1} A12
    TriSolve t{A, ld, n, A, ld, n, n, c0 + nleft, nright};
    B2M_TRY(trsm_lower_rec(ctx, st, t, c0, c0, nleft));
    // A22 -= A21 * A12
    const int64_t r1 = c0 + nleft;
    DOperand a{A, ld, n, n, r1, c0, true};
    DOperand b{A, ld, n, n, c0, r1, false};
    B2M_TRY(dgemm_tiled(ctx, st, a, b, A + r1 * ld + r1, ld, n - r1, nright, nleft, B2M_DO_SUB, true));
    return lu_rec(ctx, st, A, ld, n, r1, nright, ipiv, perm, leaf, sc);
}

constexpr int64_t kOuterNB = 256;  // outer panel width of the blocked FP64 LU
static_assert(kOuterNB == kTpK, "the panel triangular solve holds one outer panel's rows");

// Blocked right-looking LU with look-ahead (orders n > kSmallLu).  Per outer panel of 256
// columns: (1) the panel is factored right-looking by leaves, each leaf's interchanges kept inside
// the panel (and recorded in the row map pmap), its U12 and its rank-w update applied to the rest of
// the panel (to the next leaf by that leaf's own kernel, beyond it by leaf_side_kernel and
// panel_rank_update_kernel; leaves of 16 or 8 columns by leaf_swap_u12_kernel and
// panel_rank_update_kernel); (2) the
// panel's net permutation is applied to the next panel's columns on this stream, and to every
// further column right of the panel and the factored columns left of it on the side stream;
// (3) U12 = L11^-1 A12 (trsm_panel_kernel, one launch) and A22 -= A21 U12 for the next panel's
// 256 columns on this stream;
// (4) the same for every further column on the side stream, where it overlaps the next panel's
// factorisation (which reads and writes only the next panel's columns) and is joined before the
// next step's permutation moves rows under it.  The row map alternates between two buffers by panel
// parity, because the side stream may still read one panel's map while the next panel fills its own.
// Every interchange reaches every column exactly once and in order, so the factors and the pivot
// vector are those of the unblocked recursion.
// part 0 issues the first outer panel's leaves only, part 1 everything after them (two graphs: the
// device factors the first panel while the host submits the second).
int32_t lu_blocked(Ctx* ctx, cudaStream_t q, double* A, int64_t ld, int64_t n, int32_t* ipiv, int32_t* perm,
                   int32_t* pmap2, int64_t leaf, int part) {
    const bool linked = leaf == kPanelW;  // (the narrower leaves of taller matrices are not linked)
    int32_t* moves = pmap2 + 2 * round_up(n, 64);
    cudaStream_t q2 = ctx->side_stream;
    bool side_busy = false;
    auto join = [&]() -> int32_t {
        if (!side_busy) return B2M_OK;
        B2M_CU(ctx, cudaEventRecord(ctx->ev_side_join, q2));
        B2M_CU(ctx, cudaStreamWaitEvent(q, ctx->ev_side_join, 0));
        side_busy = false;
        return B2M_OK;
    };
    auto fork = [&]() -> int32_t {
        B2M_CU(ctx, cudaEventRecord(ctx->ev_side_fork, q));
        B2M_CU(ctx, cudaStreamWaitEvent(q2, ctx->ev_side_fork, 0));
        side_busy = true;
        return B2M_OK;
    };
    const int64_t pm_ld = round_up(n, 64);
    PriorityScope hi(ctx, true);  // this stream's launches are the critical path (see launch_k)
    for (int64_t k0 = 0; k0 < n; k0 += kOuterNB) {
        const int64_t w = std::min(kOuterNB, n - k0), k1 = k0 + w;
        int32_t* pmap = pmap2 + ((k0 / kOuterNB) & 1) * pm_ld;
        const bool leaves = (part == 0) == (k0 == 0);
        if (leaves) {
            B2M_CU(ctx, launch_k(ctx, iota_kernel, dim3((unsigned)ceil_div(n, 256)), dim3(256), 0, q, pmap, n));
            B2M_LAUNCHED(ctx);
        }
        // The panel, right-looking by leaves.  The critical path, on this stream: a leaf's panel
        // kernel, then its interchanges, U12 and rank-w update on the next leaf's columns only (in the
        // next leaf's own kernel when the leaves are linked); the same for the other columns of the
        // outer panel (the factored ones left of the leaf get the interchanges only) runs on the leaf stream, under the next leaf's panel kernel, and is
        // waited for before that leaf's own updates touch those columns.  Column groups are
        // disjoint between the two streams, and every column sees the leaves' interchanges and
        // updates in leaf order, so the factors are those of the single-stream order.
        cudaStream_t ql = ctx->leaf_stream;
        bool leaf_busy = false;
        auto swap_u12 = [&](cudaStream_t qs, int64_t c0, int64_t wl, int64_t lo, int64_t hi, bool maps) -> int32_t {
            const int64_t cols = std::max<int64_t>(0, (lo >= c0 + wl || hi <= c0) ? hi - lo : hi - lo - wl);
            if (cols == 0 && !maps) return B2M_OK;  // (the maps' update runs even without columns)
            prof_begin(ctx, qs, kClsSwap);
            B2M_CU(ctx, launch_k(ctx, leaf_swap_u12_kernel<double>,
                                 dim3((unsigned)std::max<int64_t>(1, ceil_div(cols, kSuThreads))),
                                 dim3(kSuThreads), 0, qs, A, ld, (int)lo, (int)hi, (int)c0, (int)wl, ipiv,
                                 maps ? perm : (int32_t*)nullptr, maps ? pmap : (int32_t*)nullptr,
                                 (const int32_t*)ctx->d_status));
            prof_end(ctx, qs, kClsSwap, 16.0 * wl * (double)cols);
            B2M_LAUNCHED(ctx);
            return B2M_OK;
        };
        auto rank_update = [&](cudaStream_t qs, int64_t c0, int64_t wl, int64_t cl, int64_t ch, int max_ctas) -> int32_t {
            const int64_t rl = c0 + wl;
            if (ch <= cl || rl >= n) return B2M_OK;
            const int64_t tiles = ceil_div(ch - cl, kRuT) * ceil_div(n - rl, kRuT);
            prof_begin(ctx, qs, kClsGemm);
            B2M_CU(ctx, launch_k(ctx, panel_rank_update_kernel<false>, dim3((unsigned)std::min<int64_t>(tiles, max_ctas)),
                                 dim3(256), 0, qs, A, ld, (int)n, (int)rl, (int)cl, (int)ch, (int)c0, (int)wl,
                                 (const int32_t*)ctx->d_status));
            prof_end(ctx, qs, kClsGemm, 2.0 * (double)(n - rl) * (double)(ch - cl) * (double)wl);  // flops
            B2M_LAUNCHED(ctx);
            return B2M_OK;
        };
        for (int64_t c0 = k0; leaves && c0 < k1; c0 += leaf) {
            const int64_t wl = std::min(leaf, k1 - c0);
            // a linked leaf applies the leaf before it to its own columns; the leaf stream does it for
            // the rest of the panel and keeps the maps
            int32_t* mv = moves + kPanelMoves * (c0 / kPanelW & 1);
            PanelLink link;
            if (linked && c0 > k0) link.moves_in = moves + kPanelMoves * ((c0 / kPanelW - 1) & 1);
            if (linked) link.moves_out = mv;
            B2M_TRY(launch_panel<double>(ctx, q, A + c0 * ld + c0, ld, (int)(n - c0), (int)wl, (int)c0, (int)c0, ipiv,
                                         link));
            const int64_t rl = c0 + wl, nx = std::min(rl + leaf, k1);  // the next leaf: columns [rl, nx)
            B2M_CU(ctx, cudaEventRecord(ctx->ev_leaf_panel, q));
            if (leaf_busy) {  // the previous leaf's updates of [rl, k1) are done
                B2M_CU(ctx, cudaStreamWaitEvent(q, ctx->ev_leaf_side, 0));
                leaf_busy = false;
            }
            if (!linked) {
                B2M_TRY(swap_u12(q, c0, wl, rl, nx, true));
                B2M_TRY(rank_update(q, c0, wl, rl, nx, 1 << 30));
            }
            if (nx < k1 || c0 > k0 || linked) {
                PriorityScope side(ctx, false);
                B2M_CU(ctx, cudaStreamWaitEvent(ql, ctx->ev_leaf_panel, 0));
                if (linked) {
                    const int64_t groups = ceil_div(c0 - k0, kPanelW) + ceil_div(k1 - nx, kPanelW);
                    prof_begin(ctx, ql, kClsSwap);
                    B2M_CU(ctx, launch_k(ctx, leaf_side_kernel, dim3((unsigned)std::max<int64_t>(1, groups)),
                                         dim3(kLsThreads), 0, ql, A, ld, (int)c0, (int)wl, (int)k0, (int)nx, (int)k1,
                                         (const int32_t*)mv, perm, pmap, (const int32_t*)ctx->d_status));
                    prof_end(ctx, ql, kClsSwap, 16.0 * wl * (double)(k1 - nx + c0 - k0));
                    B2M_LAUNCHED(ctx);
                } else {
                    B2M_TRY(swap_u12(ql, c0, wl, nx, k1, false));
                    B2M_TRY(swap_u12(ql, c0, wl, k0, c0, false));
                }
                // (the next leaf's cluster needs 16 SMs to itself)
                B2M_TRY(rank_update(ql, c0, wl, nx, k1, linked ? 2 * (ctx->num_sms - 16) : 64));
                B2M_CU(ctx, cudaEventRecord(ctx->ev_leaf_side, ql));
                leaf_busy = true;
            }
            B2M_TRY(report_progress(ctx, q, c0 + wl, n));
        }
        if (leaf_busy) B2M_CU(ctx, cudaStreamWaitEvent(q, ctx->ev_leaf_side, 0));
        if (part == 0) return B2M_OK;
        B2M_TRY(join());  // the previous panel's wide update is done before rows move under it
        auto permute = [&](cudaStream_t qs, int64_t c_begin, int64_t c_end) -> int32_t {
            if (c_end <= c_begin) return B2M_OK;
            prof_begin(ctx, qs, kClsSwap);
            B2M_CU(ctx, launch_k(ctx, panel_permute_f64_kernel, dim3((unsigned)ceil_div(c_end - c_begin, 32)), dim3(256), 0,
                                 qs, A, ld, (int)n, (int)k0, (int)c_begin, (int)c_end, (const int32_t*)pmap,
                                 ctx->d_status));
            prof_end(ctx, qs, kClsSwap, 2.0 * 8.0 * 2 * w * (double)(c_end - c_begin));  // <= 2w rows moved
            B2M_LAUNCHED(ctx);
            return B2M_OK;
        };
        const int64_t rest = n - k1, nw = std::min(kOuterNB, std::max<int64_t>(rest, 0));
        // only the next panel's columns are permuted on this stream; the other columns right of
        // the panel and the factored columns left of it on the side stream, ahead of their update
        B2M_TRY(permute(q, k1, k1 + nw));
        if (k0 > 0 || rest > nw) {
            B2M_TRY(fork());
            PriorityScope side(ctx, false);
            B2M_TRY(permute(q2, k1 + nw, n));
            B2M_TRY(permute(q2, 0, k0));
        }
        if (k1 >= n) break;
        auto update = [&](cudaStream_t qs, int64_t cs, int64_t nc) -> int32_t {
            B2M_TRY(launch_trsm_panel(ctx, qs, A + k0 * ld + k0, ld, A + k0 * ld + cs, ld, (int)w, nc, false));
            DOperand a{A, ld, n, n, k1, k0, true};
            DOperand b{A, ld, n, n, k0, cs, false};
            return dgemm_tiled(ctx, qs, a, b, A + k1 * ld + cs, ld, n - k1, nc, w, B2M_DO_SUB, true);
        };
        if (rest > nw) {
            PriorityScope side(ctx, false);
            B2M_TRY(update(q2, k1 + nw, rest - nw));
        }
        B2M_TRY(update(q, k1, nw));
    }
    return join();
}


}  // namespace

// the low-priority side stream (and its fork/join events) of this context, created on first use
int32_t ensure_side_stream(Ctx* ctx) {
    if (ctx->side_stream && ctx->leaf_stream) return B2M_OK;
    int least = 0, greatest = 0;
    B2M_CU(ctx, cudaDeviceGetStreamPriorityRange(&least, &greatest));
    if (!ctx->side_stream) {
        B2M_CU(ctx, cudaStreamCreateWithPriority(&ctx->side_stream, cudaStreamNonBlocking, least));
        B2M_CU(ctx, cudaEventCreateWithFlags(&ctx->ev_side_fork, cudaEventDisableTiming));
        B2M_CU(ctx, cudaEventCreateWithFlags(&ctx->ev_side_join, cudaEventDisableTiming));
    }
    // the FP64 LU's in-panel look-ahead: the stream runs at the critical path's priority, since the
    // leaf after next waits for it
    B2M_CU(ctx, cudaStreamCreateWithPriority(&ctx->leaf_stream, cudaStreamNonBlocking, greatest));
    B2M_CU(ctx, cudaEventCreateWithFlags(&ctx->ev_leaf_panel, cudaEventDisableTiming));
    B2M_CU(ctx, cudaEventCreateWithFlags(&ctx->ev_leaf_side, cudaEventDisableTiming));
    ctx->chain_priority = greatest;
    return B2M_OK;
}

int32_t chol_panel_update(Ctx* ctx, cudaStream_t st, double* A, int64_t ld, int64_t n, int64_t c0, int64_t cl,
                          int64_t ch) {
    if (ch <= cl) return B2M_OK;
    const int64_t tiles = ceil_div(ch - cl, kRuT) * ceil_div(n - cl, kRuT);
    prof_begin(ctx, st, kClsGemm);
    B2M_CU(ctx, launch_k(ctx, panel_rank_update_kernel<true>, dim3((unsigned)tiles), dim3(256), 0, st, A, ld, (int)n,
                         (int)cl, (int)cl, (int)ch, (int)c0, kPanelW, (const int32_t*)ctx->d_status));
    prof_end(ctx, st, kClsGemm, 2.0 * (double)(n - cl) * (double)(ch - cl) * kPanelW);  // flops
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

template <typename T>
int32_t launch_swaps(Ctx* ctx, cudaStream_t st, T* A, int64_t ld, int ncols, int c0, int w, const int32_t* ipiv,
                     int32_t* perm) {
    return launch_swaps_impl<T>(ctx, st, A, ld, ncols, c0, w, ipiv, perm);
}
template int32_t launch_swaps<double>(Ctx*, cudaStream_t, double*, int64_t, int, int, int, const int32_t*, int32_t*);

int32_t lu_factor_f64(Ctx* ctx, cudaStream_t st, double* A, int64_t ld, int64_t n, int32_t* ipiv, int32_t* perm) {
    if (n <= 0) return B2M_OK;
    if ((ld & 1) || !aligned16(A)) return fail(ctx, B2M_ERR_DIM, "lu_factor_f64: ld must be even, A 16-byte aligned");
    if (n > (1 << 30)) return fail(ctx, B2M_ERR_UNSUPPORTED, "n too large");
    // the leaf width shrinks as the first panel grows (the cluster holds a whole panel on chip)
    const int64_t leaf = n <= panel_max_rows(true, 32) ? 32 : (n <= panel_max_rows(true, 16) ? 16 : 8);
    if (n > panel_max_rows(true, 8))
        return fail(ctx, B2M_ERR_UNSUPPORTED, "FP64 LU supports n <= %d", panel_max_rows(true, 8));
    if (ctx->progress) {
        // the notes are the host functions' payloads: wait until the previous call's have run, then
        // reserve one per leaf so that none moves while queued
        B2M_CU(ctx, cudaStreamSynchronize(st));
        ctx->progress_notes.clear();
        ctx->progress_notes.reserve((size_t)(n / 8 + 2));
    }
    // Three ways, by the order (measured, factor + solve of one right-hand side, us):
    //   * up to 256 (kSmallLu), one launch of one CTA (order 16: 33 against 44 by the recursion, 100: 125 / 201,
    //     256: 339 / 429 and about 375 by the blocked driver);
    //   * above, the blocked look-ahead driver with linked leaves (257: 366 / 491, 512: 652 / 931);
    //   * the plain recursion where no workspace or side stream may be used (the allocation-free entry
    //     point, n <= 512).
    // Every order asks for the small orders' scratch and the side streams, so that after a call of any order
    // a smaller one allocates nothing (and can be captured).
    const bool plain = ctx->fixed_scratch;
    const bool blocked = !plain && n > kSmallLu;
    void* scratch = nullptr;
    if (!ctx->fixed_scratch) {
        const size_t maps = (size_t)(2 * round_up(n, 64) + 2 * kPanelMoves) * sizeof(int32_t);
        B2M_TRY(ws_get(ctx, kWsPmap, std::max(maps, small_lu_scratch(kSmallLu)), &scratch));
        B2M_TRY(ensure_side_stream(ctx));
    }
    if (!plain && !blocked) {
        B2M_TRY(small_lu_f64(ctx, st, A, ld, n, static_cast<double*>(scratch), ipiv, perm));
        for (int64_t c = 0; ctx->progress && c < n; c += leaf)
            B2M_TRY(report_progress(ctx, st, std::min(n, c + leaf), n));
        return B2M_OK;
    }
    int32_t* pmap2 = static_cast<int32_t*>(scratch);
    const GraphKey key{1, A, ipiv, perm, ctx->d_status, ld, n, 0, 0};
    const GraphKey key1{1, A, ipiv, perm, ctx->d_status, ld, n, 0, 1};
    B2M_TRY(run_graph(ctx, st, key, [&](cudaStream_t s) -> int32_t {
        if (perm) {
            iota_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(perm, n);
            B2M_LAUNCHED(ctx);
        }
        if (blocked) return lu_blocked(ctx, s, A, ld, n, ipiv, perm, pmap2, leaf, 0);
        return lu_rec(ctx, s, A, ld, n, 0, n, ipiv, perm, leaf, SwapScope{0, n, nullptr});
    }));
    if (!blocked) return B2M_OK;
    return run_graph(ctx, st, key1, [&](cudaStream_t s) -> int32_t {
        return lu_blocked(ctx, s, A, ld, n, ipiv, perm, pmap2, leaf, 1);
    });
}

int32_t lu_solve_f64(Ctx* ctx, cudaStream_t st, const double* LU, int64_t ld, int64_t n, const int32_t* perm,
                     double* B, int64_t ldb, int64_t nrhs, double* tmp) {
    if (n <= 0 || nrhs <= 0) return B2M_OK;
    if ((ldb & 1) || !aligned16(B)) return fail(ctx, B2M_ERR_DIM, "lu_solve_f64: ldb must be even");
    // (order 16, one right-hand side: 18 us against 23 by a copy, a gather and two sweeps, 100: 40 / 50, 256: 79 / 89;
    // 256 right-hand sides 91 / 212)
    if (n <= kSmallLu) return small_solve_f64(ctx, st, LU, ld, n, perm, B, ldb, nrhs);
    // X = P B
    double* X = tmp;
    if (!X) {
        void* w = nullptr;
        B2M_TRY(ws_get(ctx, kWsE, (size_t)(n * ldb * sizeof(double)), &w));
        X = static_cast<double*>(w);
    }
    const GraphKey key{2, LU, perm, B, X, ld, n, ldb, nrhs};
    return run_graph(ctx, st, key, [&](cudaStream_t s) -> int32_t {
        B2M_CU(ctx, cudaMemcpy2DAsync(X, ldb * 8, B, ldb * 8, nrhs * 8, n, cudaMemcpyDeviceToDevice, s));
        gather_rows_kernel<<<(unsigned)ceil_div(n * nrhs, 256), 256, 0, s>>>(B, ldb, X, ldb, perm, n, nrhs);
        B2M_LAUNCHED(ctx);
        // few right-hand sides: block-row sweeps (dtrsv.cu), whose workspace and side stream the allocation-free
        // entry point may not ask for
        if (nrhs <= 64 && !ctx->fixed_scratch) {
            return tri_solve2_f64(ctx, s, LU, ld, n, kTriL, kTriU, B, ldb, nrhs);
        }
        TriSolve t{LU, ld, n, B, ldb, n, nrhs, 0, nrhs};
        B2M_TRY(trsm_lower_rec(ctx, s, t, 0, 0, n));
        return trsm_upper_rec(ctx, s, t, 0, 0, n);
    });
}

int32_t perm_from_ipiv(Ctx* ctx, cudaStream_t st, const int32_t* ipiv, int64_t n, int32_t* perm) {
    if (n > (1 << 30)) return fail(ctx, B2M_ERR_UNSUPPORTED, "perm_from_ipiv: n too large");
    const size_t smem = (size_t)n * 3 * sizeof(uint16_t);
    if (n <= kPermMax && smem <= ctx->smem_optin) {
        std::atomic<int>& set = device_flag((const void*)perm_from_ipiv_kernel, 0, ctx->device);
        if (!set.load()) {
            B2M_CU(ctx, cudaFuncSetAttribute(perm_from_ipiv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             3 * kPermMax * (int)sizeof(uint16_t)));
            set.store(1);
        }
        perm_from_ipiv_kernel<<<1, kPermThreads, smem, st>>>(ipiv, (int)n, perm);
    } else {
        const size_t copy = (size_t)n * sizeof(int32_t);
        const bool in_smem = copy <= ctx->smem_optin;
        std::atomic<int>& set = device_flag((const void*)perm_from_ipiv_serial_kernel, 0, ctx->device);
        if (in_smem && !set.load()) {
            B2M_CU(ctx, cudaFuncSetAttribute(perm_from_ipiv_serial_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)ctx->smem_optin));
            set.store(1);
        }
        perm_from_ipiv_serial_kernel<<<1, 1024, in_smem ? copy : 0, st>>>(ipiv, (int)n, perm, in_smem ? 1 : 0);
    }
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t lu_determinant(Ctx* ctx, cudaStream_t st, const double* LU, int64_t ld, int64_t n, const int32_t* ipiv,
                       double* d_det) {
    if (n > (1 << 30)) return fail(ctx, B2M_ERR_UNSUPPORTED, "determinant: n too large");
    determinant_kernel<<<1, kDetChunk, 0, st>>>(LU, ld, (int)n, ipiv, ctx->d_status, d_det);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

// A strided copy of doubles, by pairs (T = double2) where both sides allow it.  Bound by HBM / L2; a
// thread moves kCopyRows elements of one column so that their loads are in flight together.  Repacking
// an 8191 x 8191 matrix (rows of odd length) takes 153 us (7.0 TB/s), a 2999 x 1501 one 10 us;
// cudaMemcpy2DAsync took 544 and 41 us.
constexpr int kCopyRows = 8;
template <typename T>
__global__ void __launch_bounds__(256) copy_matrix_kernel(T* dst, int64_t ldd, const T* src, int64_t lds, int rows,
                                                          int cols) {
    const int c = blockIdx.x * 64 + (threadIdx.x & 63);
    const int r0 = blockIdx.y * 4 * kCopyRows + (threadIdx.x >> 6);
    if (c >= cols) return;
    T v[kCopyRows];
#pragma unroll
    for (int i = 0; i < kCopyRows; ++i)
        if (r0 + 4 * i < rows) v[i] = src[(int64_t)(r0 + 4 * i) * lds + c];
#pragma unroll
    for (int i = 0; i < kCopyRows; ++i)
        if (r0 + 4 * i < rows) dst[(int64_t)(r0 + 4 * i) * ldd + c] = v[i];
}

int32_t copy_matrix(Ctx* ctx, cudaStream_t st, double* dst, int64_t ldd_bytes, const double* src, int64_t lds_bytes,
                    int64_t rows, int64_t cols) {
    if (rows <= 0 || cols <= 0) return B2M_OK;
    const int64_t gy = ceil_div(rows, 4 * kCopyRows);
    if (gy > 65535 || cols > (1 << 30)) {  // beyond the launch grid
        B2M_CU(ctx, cudaMemcpy2DAsync(dst, ldd_bytes, src, lds_bytes, cols * 8, rows, cudaMemcpyDeviceToDevice, st));
        return B2M_OK;
    }
    if (aligned16(dst) && aligned16(src) && ((ldd_bytes | lds_bytes) & 15) == 0 && cols % 2 == 0)
        copy_matrix_kernel<double2><<<dim3((unsigned)ceil_div(cols / 2, 64), (unsigned)gy), 256, 0, st>>>(
            reinterpret_cast<double2*>(dst), ldd_bytes / 16, reinterpret_cast<const double2*>(src), lds_bytes / 16,
            (int)rows, (int)(cols / 2));
    else
        copy_matrix_kernel<double><<<dim3((unsigned)ceil_div(cols, 64), (unsigned)gy), 256, 0, st>>>(
            dst, ldd_bytes / 8, src, lds_bytes / 8, (int)rows, (int)cols);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

}  // namespace b2m

namespace b2m {

__global__ void axpy_matrix_kernel(double* X, int64_t ldx, const double* R, int64_t ldr, int64_t rows, int64_t cols,
                                   const int32_t* status) {
    if (status[kInfo] != 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= rows * cols) return;
    const int64_t i = e / cols, c = e - i * cols;
    X[i * ldx + c] += R[i * ldr + c];
}

__global__ void set_diagonal_kernel(double* X, int64_t ldx, int64_t n, double v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) X[i * ldx + i] = v;
}

__global__ void copy_if_ok_kernel(double* dst, int64_t ldd, const double* src, int64_t lds, int64_t rows, int64_t cols,
                                  const int32_t* status) {
    if (status[kInfo] != 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= rows * cols) return;
    const int64_t i = e / cols, c = e - i * cols;
    dst[i * ldd + c] = src[i * lds + c];
}

__global__ void publish_status_kernel(const int32_t* words, int32_t* out) {
    *out = words[kTimeout] != 0 ? B2M_ERR_TIMEOUT : words[kInfo];
}

int32_t publish_status(Ctx* ctx, cudaStream_t st, const int32_t* words, int32_t* out) {
    publish_status_kernel<<<1, 1, 0, st>>>(words, out);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t axpy_matrix(Ctx* ctx, cudaStream_t st, double* X, int64_t ldx, const double* R, int64_t ldr, int64_t rows,
                    int64_t cols) {
    if (rows <= 0 || cols <= 0) return B2M_OK;
    axpy_matrix_kernel<<<(unsigned)ceil_div(rows * cols, 256), 256, 0, st>>>(X, ldx, R, ldr, rows, cols,
                                                                             ctx->d_status);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t set_diagonal(Ctx* ctx, cudaStream_t st, double* X, int64_t ldx, int64_t n, double v) {
    if (n <= 0) return B2M_OK;
    set_diagonal_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(X, ldx, n, v);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t copy_if_ok(Ctx* ctx, cudaStream_t st, double* dst, int64_t ldd, const double* src, int64_t lds, int64_t rows,
                   int64_t cols) {
    if (rows <= 0 || cols <= 0) return B2M_OK;
    copy_if_ok_kernel<<<(unsigned)ceil_div(rows * cols, 256), 256, 0, st>>>(dst, ldd, src, lds, rows, cols,
                                                                           ctx->d_status);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

}  // namespace b2m
