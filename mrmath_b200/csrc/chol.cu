// chol.cu -- Cholesky factorisation A = L L^T of a symmetric positive-definite FP64 matrix and the
// solve built on it (the next dense factorisation on the LU path's DGEMM and triangular sweeps).
//
// Reference: TDoubleMatrix.Cholesky (DblMatrix.pas:967-990) -> MatrixCholeskyInPlace4
// (LinAlgCholesky.pas:106-123), a left-looking blocked Cholesky with 32-column panels
// (InternalBlkCholeskyInPlace :54-103: rank-k update of the diagonal block, unblocked factorisation
// MatrixCholeskyInPlace2 :205-250, MultT2 update of the column below, triangular solve with the
// reciprocal of each diagonal element); the Numerical-Recipes form MatrixCholeskyInPlace (:270-332,
// L below the diagonal, its diagonal in a separate vector P) and MatrixCholeskySolveLinEq
// (:352-421).  Result: 0 = crOk, 1 = crNoPositiveDefinite (MatrixConst.pas:30) when a diagonal
// element is <= 0 or NaN before its square root.
//
// B200 design: outer panels of 256 columns, right-looking.  What bounds it is the chain of the
// columns (a square root, a division and a row of products each), so a 32-column leaf is one kernel:
// chol_leaf_kernel applies the previous leaf's 32 columns to the leaf, then eliminates, every CTA
// carrying its own copy of the leaf's 32 x 32 diagonal block beside its 64 rows (no grid-wide wait).
// The other columns of the panel get a leaf's update on the leaf stream, under the next leaf.  After
// a panel, the next panel's columns get its K = 256 update on this stream and the rest of the
// trailing lower triangle on the side stream (look-ahead), in one product whose tiles above the
// diagonal return at once.  The factorisation runs on a workspace copy, so the caller's strict upper
// triangle is never written.
#include <cfloat>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace b2m {
namespace {

constexpr int kChLeaf = 32;        // leaf width
constexpr int kChPanel = 256;      // outer panel width
constexpr int kChRows = 64;        // rows per leaf CTA
constexpr int kChThreads = (kChLeaf + kChRows) * kChLeaf / 16;  // 4 x 4 elements a thread
constexpr int kChPitch = kChLeaf + 1;

// Root and reciprocal root of p by Goldschmidt's coupled iteration from the approximate reciprocal
// root: g -> sqrt(p), h -> 1 / (2 sqrt(p)), two steps (2^-22 -> 2^-44 -> rounding), then one
// correction of g by its exact residual p - g g, which leaves it within an ulp of sqrt(p).  Straight
// code, so that the row updates of the column before run under it; sqrt and a division took 246
// cycles of a column's chain.
__device__ __forceinline__ void chol_root(double p, double& d, double& y) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(p));
    double g = p * y0, h = 0.5 * y0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double r = fma(-g, h, 0.5);
        g = fma(g, r, g);
        h = fma(h, r, h);
    }
    d = fma(fma(-g, g, p), h, g);
    y = h + h;
}
// where no step of chol_root can leave the normal numbers
__device__ __forceinline__ bool chol_in_range(double p) { return p > 1e-250 && p < 1e250; }
// x / d: the product with the reciprocal, corrected by its exact residual; y = 0 asks for a division
__device__ __forceinline__ double chol_quot(double x, double d, double y) {
    if (__double2hiint(y) == 0) return x / d;
    const double q = x * y;
    return fma(fma(-q, d, x), y, q);
}

// Leaf [c, c + w) of the n x n matrix (row stride ld), w <= 32.  pc >= 0: the 32 columns [pc, c) of
// the leaf before, whose update these columns still lack (every older one is in).  Thread t < 96 of
// CTA b then owns one row: t < 32 row c + t of the diagonal block, else row c + 32 + 64 b + t - 32.
//
// All rows are eliminated together, a column at a time: warp 0 takes the square root of the diagonal
// element, every row divides its element by it, warp 0's quotients go to shared memory (one barrier)
// and every row subtracts its multiple of them; rows shift left by one, so register indices are
// compile-time in a compact loop body, in four phases as the rows get shorter.  The next column is
// updated first, and its root runs under the rest.  The diagonal block of L goes to
// `diag` (n x 32), because other CTAs may still be reading the block itself.
//
// Measured on a B200 at 3000 rows: 200 us and 46 us of a separate product before (a fully unrolled
// 32 x 32 elimination and panels read row by row), now about 11 us with the update; the factor and a
// solve of order 3000 together 21.97 -> 1.92 ms.
__global__ void __launch_bounds__(kChThreads) chol_leaf_kernel(double* A, int64_t ld, int n, int c, int w, int pc,
                                                               double* diag, int32_t* status) {
    __shared__ double s_p[kChLeaf + kChRows][kChPitch];  // the previous leaf's rows, then this leaf's
    __shared__ double s_c[2][2 * kChLeaf];               // column of L11, by parity, zero past its end
    __shared__ double2 s_d[2];                           // (root, 1 / root) of the diagonal element
    __shared__ int s_bad;
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31;
    const int r0 = c + kChLeaf + blockIdx.x * kChRows;
    auto row_of = [&](int i) { return i < kChLeaf ? c + i : r0 + i - kChLeaf; };
    auto valid = [&](int i) { return i < kChLeaf ? i < w : r0 + i - kChLeaf < n; };
    if (t == 0) s_bad = 0;
    if (t < 2 * kChLeaf) s_c[0][t] = s_c[1][t] = 0.0;
    // this thread's 4 x 4 elements of the leaf, and the previous leaf's rows
    const int ty = t >> 3, tx = t & 7;
    double x[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            x[i][j] = (valid(4 * ty + i) && 4 * tx + j < w) ? A[(int64_t)row_of(4 * ty + i) * ld + c + 4 * tx + j] : 0.0;
    if (pc >= 0) {
        batched_copy<kChThreads, (kChLeaf + kChRows) * kChLeaf / kChThreads, double>(t, (kChLeaf + kChRows) * kChLeaf,
            [&](int e) { return valid(e >> 5) ? A[(int64_t)row_of(e >> 5) * ld + pc + (e & 31)] : 0.0; },
            [&](int e, double v) { s_p[e >> 5][e & 31] = v; });
        __syncthreads();
        double acc[4][4] = {};
#pragma unroll 4
        for (int k = 0; k < kChLeaf; ++k) {
            double av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = s_p[4 * ty + i][k];
#pragma unroll
            for (int j = 0; j < 4; ++j) bv[j] = s_p[4 * tx + j][k];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) x[i][j] -= acc[i][j];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s_p[4 * ty + i][4 * tx + j] = x[i][j];
    __syncthreads();
    constexpr int kOwners = kChLeaf + kChRows;
    if (t < kOwners) {
        double r[kChLeaf];
#pragma unroll
        for (int k = 0; k < kChLeaf; ++k) r[k] = (t >= kChLeaf || k <= t) ? s_p[t][k] : 0.0;
        double d = 1.0, y = 1.0;  // warp 0: the root of the next diagonal element and its reciprocal
        bool bad = false;         // warp 0: a diagonal element was <= 0 or NaN (the rest is then not used)
        auto root = [&](double p) {
            bad = bad || !(p > 0.0);
            if (!chol_in_range(p)) {
                d = p > 0.0 ? sqrt(p) : 1.0;
                y = 0.0;
            }
        };
        if (t < kChLeaf) {
            const double p = __shfl_sync(0xffffffffu, r[0], 0);
            chol_root(p, d, y);
            root(p);
        }
        // columns [j0, j0 + 8), kLen the row length at j0
        auto phase = [&](const int j0, auto len) {
            constexpr int kLen = decltype(len)::value;
#pragma unroll 1
            for (int j = j0; j < min(j0 + 8, w); ++j) {
                const int par = j & 1;
                const double* lc = &s_c[par][j];
                if (t < kChLeaf) {  // warp 0
                    const double q = chol_quot(lane > j ? r[0] : d, d, y);
                    const double l = lane > j ? q : (lane == j ? d : 0.0);
                    s_c[par][lane] = l;
                    if (lane == 0) s_d[par] = make_double2(d, y);
                    asm volatile("bar.sync 1, %0;\n" ::"n"(kOwners) : "memory");
                    r[0] = fma(-l, lc[1], r[1]);
                    const double p = __shfl_sync(0xffffffffu, r[0], (j + 1) & 31);
                    chol_root(p, d, y);
#pragma unroll
                    for (int k = 2; k < kLen; ++k) r[k - 1] = fma(-l, lc[k], r[k]);
                    s_p[t][j] = l;
                    if (j + 1 < w) root(p);
                } else {
                    asm volatile("bar.sync 1, %0;\n" ::"n"(kOwners) : "memory");
                    const double2 dy = s_d[par];
                    const double l = chol_quot(r[0], dy.x, dy.y);
                    s_p[t][j] = l;
#pragma unroll
                    for (int k = 1; k < kLen; ++k) r[k - 1] = fma(-l, lc[k], r[k]);
                }
                r[kLen - 1] = 0.0;
            }
        };
        phase(0, std::integral_constant<int, 32>{});
        phase(8, std::integral_constant<int, 24>{});
        phase(16, std::integral_constant<int, 16>{});
        phase(24, std::integral_constant<int, 8>{});
        if (bad) s_bad = 1;
    }
    __syncthreads();
    if (s_bad) {
        if (t == 0 && blockIdx.x == 0) atomicExch(&status[kInfo], 1);
        return;
    }
    // L's rows below the block; the block itself to `diag` (its strict upper part is not read)
    for (int e = t; e < kChRows * kChLeaf; e += kChThreads) {
        const int i = kChLeaf + (e >> 5), k = e & 31;
        if (valid(i) && k < w) A[(int64_t)row_of(i) * ld + c + k] = s_p[i][k];
    }
    if (blockIdx.x == 0)
        for (int e = t; e < kChLeaf * kChLeaf; e += kChThreads) {
            const int i = e >> 5, k = e & 31;
            if (i < w && k <= i) diag[(int64_t)(c + i) * kChLeaf + k] = s_p[i][k];
        }
}

// the diagonal blocks of L (n x 32 in `diag`) into A's
__global__ void chol_diag_kernel(double* A, int64_t ld, int n, const double* diag, const int32_t* status) {
    if (status[kInfo] != 0) return;
    const int e = blockIdx.x * blockDim.x + threadIdx.x, i = e / kChLeaf, k = e % kChLeaf;
    if (i < n && k <= i % kChLeaf) A[(int64_t)i * ld + i / kChLeaf * kChLeaf + k] = diag[e];
}

// dst's lower triangle (diagonal included) <- src's, when status[kInfo] == 0
__global__ void copy_lower_kernel(double* dst, int64_t ldd, const double* src, int64_t lds, int64_t n,
                                  const int32_t* status) {
    if (status && status[kInfo] != 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t i = e / n, j = e - i * n;
    if (j <= i) dst[i * ldd + j] = src[i * lds + j];
}

// W's upper triangle (diagonal included) <- the transpose of F's lower triangle: 32 x 32 tiles through
// shared memory, rows read and written whole (3000 x 3000: 11 us; a copy and an element-wise transpose
// took 31 + 20)
__global__ void __launch_bounds__(256) transpose_lower_kernel(double* W, int64_t ldw, const double* F, int64_t ldf,
                                                              int n) {
    __shared__ double tile[32][33];
    const int bi = blockIdx.y * 32, bj = blockIdx.x * 32;  // F's rows and columns
    if (bj > bi) return;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = wp + 8 * q;
        if (bi + r < n && bj + lane < n) tile[r][lane] = F[(int64_t)(bi + r) * ldf + bj + lane];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = wp + 8 * q, i = bi + lane, j = bj + r;
        if (i < n && j < n && j <= i) W[(int64_t)j * ldw + i] = tile[lane][r];
    }
}

// L's strict lower triangle and P's diagonal from one factor (NR form): Lnr[i][j] = F[i][j] (j < i),
// P[i] = F[i][i] (P element i at byte offset i * lwp)
__global__ void split_nr_kernel(double* Lnr, int64_t ldl, double* P, int64_t lwp, const double* F, int64_t ldf,
                                int64_t n, const int32_t* status) {
    if (status[kInfo] != 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t i = e / n, j = e - i * n;
    if (j < i) Lnr[i * ldl + j] = F[i * ldf + j];
    if (j == i) *reinterpret_cast<double*>(reinterpret_cast<char*>(P) + i * lwp) = F[i * ldf + i];
}

// F <- Lnr's strict lower triangle with P on the diagonal (the NR form joined into one factor)
__global__ void join_nr_kernel(double* F, int64_t ldf, const double* Lnr, int64_t ldl, const double* P, int64_t lwp,
                               int64_t n) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t i = e / n, j = e - i * n;
    if (j < i) F[i * ldf + j] = Lnr[i * ldl + j];
    if (j == i) F[i * ldf + i] = *reinterpret_cast<const double*>(reinterpret_cast<const char*>(P) + i * lwp);
}

unsigned blocks_for(int64_t e) { return (unsigned)ceil_div(std::max<int64_t>(e, 1), 256); }

}  // namespace

int32_t chol_factor_f64(Ctx* ctx, cudaStream_t st, double* A, int64_t ld, int64_t n) {
    if (n <= 0) return B2M_OK;
    if ((ld & 1) || !aligned16(A)) return fail(ctx, B2M_ERR_DIM, "chol_factor_f64: ld must be even, A 16-byte aligned");
    if (n > (1 << 30)) return fail(ctx, B2M_ERR_UNSUPPORTED, "chol_factor_f64: n too large");
    void* pd = nullptr;
    B2M_TRY(ws_get(ctx, kWsTri, (size_t)n * kChLeaf * sizeof(double), &pd));
    double* diag = static_cast<double*>(pd);
    B2M_TRY(ensure_side_stream(ctx));
    const GraphKey key{20, A, diag, nullptr, ctx->d_status, ld, n, 0, 0};
    return run_graph(ctx, st, key, [&](cudaStream_t s) -> int32_t {
        // Column groups: a leaf's kernel writes its own 32 columns; its update of the panel's columns
        // beyond the next leaf runs on the leaf stream and is waited for by the leaf after next; the
        // trailing update beyond the next panel runs on the side stream and is waited for before the
        // next panel's own trailing update.  Every column sees the updates in order.
        cudaStream_t q2 = ctx->side_stream, ql = ctx->leaf_stream;
        PriorityScope hi(ctx, true);
        bool leaf_busy = false, side_busy = false;
        for (int64_t k0 = 0; k0 < n; k0 += kChPanel) {
            const int64_t k1 = std::min(n, k0 + kChPanel);
            for (int64_t c = k0; c < k1; c += kChLeaf) {
                const int64_t w = std::min<int64_t>(kChLeaf, k1 - c), below = std::max<int64_t>(0, n - c - kChLeaf);
                prof_begin(ctx, s, kClsPanel);
                B2M_CU(ctx, launch_k(ctx, chol_leaf_kernel, dim3((unsigned)std::max<int64_t>(1, ceil_div(below, kChRows))),
                                     dim3(kChThreads), 0, s, A, ld, (int)n, (int)c, (int)w,
                                     (int)(c > k0 ? c - kChLeaf : -1), diag, ctx->d_status));
                prof_end(ctx, s, kClsPanel, 2.0 * (n - c) * w * 8.0);
                B2M_LAUNCHED(ctx);
                if (leaf_busy) B2M_CU(ctx, cudaStreamWaitEvent(s, ctx->ev_leaf_side, 0));
                leaf_busy = false;
                if (c + 2 * kChLeaf < k1) {
                    B2M_CU(ctx, cudaEventRecord(ctx->ev_leaf_panel, s));
                    B2M_CU(ctx, cudaStreamWaitEvent(ql, ctx->ev_leaf_panel, 0));
                    PriorityScope side(ctx, false);
                    B2M_TRY(chol_panel_update(ctx, ql, A, ld, n, c, c + 2 * kChLeaf, k1));
                    B2M_CU(ctx, cudaEventRecord(ctx->ev_leaf_side, ql));
                    leaf_busy = true;
                }
            }
            if (k1 >= n) break;
            if (side_busy) {  // the previous panel's update of these columns
                B2M_CU(ctx, cudaEventRecord(ctx->ev_side_join, q2));
                B2M_CU(ctx, cudaStreamWaitEvent(s, ctx->ev_side_join, 0));
                side_busy = false;
            }
            // rows and columns [cs, ...) of the trailing lower triangle -= L[., k0:k1] L[., k0:k1]^T
            auto update = [&](cudaStream_t qs, int64_t cs, int64_t nc) -> int32_t {
                DOperand a{A, ld, n, n, cs, k0, true};
                DOperand b{A, ld, n, n, cs, k0, true};
                return dgemm_tiled(ctx, qs, a, b, A + cs * ld + cs, ld, n - cs, nc, k1 - k0, B2M_DO_SUB, true, true);
            };
            const int64_t k2 = std::min(n, k1 + kChPanel);
            if (k2 < n) {
                B2M_CU(ctx, cudaEventRecord(ctx->ev_side_fork, s));
                B2M_CU(ctx, cudaStreamWaitEvent(q2, ctx->ev_side_fork, 0));
                PriorityScope side(ctx, false);
                B2M_TRY(update(q2, k2, n - k2));
                side_busy = true;
            }
            B2M_TRY(update(s, k1, k2 - k1));
        }
        chol_diag_kernel<<<blocks_for(n * kChLeaf), 256, 0, s>>>(A, ld, (int)n, diag, ctx->d_status);
        B2M_LAUNCHED(ctx);
        return B2M_OK;
    });
}

// Solves A X = B from a Cholesky factor F (lower triangle, diagonal included, row stride ldf):
// U = L^T is put into the upper triangle of the workspace W (n x ldw), then two FP64 sweeps: L y = b (the
// transposed upper triangle, true division) and L^T x = y.  B (n x nrhs, ldb) is overwritten with X.
int32_t chol_solve_f64(Ctx* ctx, cudaStream_t st, const double* F, int64_t ldf, int64_t n, double* W, int64_t ldw,
                       double* B, int64_t ldb, int64_t nrhs) {
    if (n <= 0 || nrhs <= 0) return B2M_OK;
    if (ceil_div(n, 32) > 65535) return fail(ctx, B2M_ERR_UNSUPPORTED, "chol_solve_f64: n too large");
    const unsigned nt = (unsigned)ceil_div(n, 32);
    transpose_lower_kernel<<<dim3(nt, nt), 256, 0, st>>>(W, ldw, F, ldf, (int)n);
    B2M_LAUNCHED(ctx);
    return tri_solve2_f64(ctx, st, W, ldw, n, kTriUt, kTriU, B, ldb, nrhs);
}

int32_t copy_lower(Ctx* ctx, cudaStream_t st, double* dst, int64_t ldd, const double* src, int64_t lds, int64_t n,
                   bool only_if_ok) {
    if (n <= 0) return B2M_OK;
    copy_lower_kernel<<<blocks_for(n * n), 256, 0, st>>>(dst, ldd, src, lds, n, only_if_ok ? ctx->d_status : nullptr);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t split_nr(Ctx* ctx, cudaStream_t st, double* Lnr, int64_t ldl, double* P, int64_t lwp, const double* F,
                 int64_t ldf, int64_t n) {
    if (n <= 0) return B2M_OK;
    split_nr_kernel<<<blocks_for(n * n), 256, 0, st>>>(Lnr, ldl, P, lwp, F, ldf, n, ctx->d_status);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t join_nr(Ctx* ctx, cudaStream_t st, double* F, int64_t ldf, const double* Lnr, int64_t ldl, const double* P,
                int64_t lwp, int64_t n) {
    if (n <= 0) return B2M_OK;
    join_nr_kernel<<<blocks_for(n * n), 256, 0, st>>>(F, ldf, Lnr, ldl, P, lwp, n);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

}  // namespace b2m
