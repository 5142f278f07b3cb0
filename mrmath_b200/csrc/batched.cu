// batched.cu -- many independent LU solves of uneven order in one persistent launch.
//
// There is no counterpart in the reference, which solves one system per MatrixLinEQSolve call
// (LinAlgLU.pas:481-592); every system here follows that routine's semantics: partial pivoting with
// the first maximum winning, the pivot column scaled by the reciprocal of the pivot, a pivot of
// magnitude <= 10/MaxDouble reporting the system singular (:246-268), forward substitution with the
// unit-lower factor and back substitution dividing by U's diagonal (:315-385).
//
// The host sorts the systems largest first; resident CTAs pull them from an atomic work queue
// (longest-processing-time first, no tail of big systems).
//
// Mode 0 (FP64): see batch_lu_kernel.
//
// Mode 1: systems of order > small_n take a whole CTA; smaller ones are handed out in batches, one per
// group of G warps, each group with its own named barrier.  The panel width of both size buckets and G
// are chosen by the autotuner at the bottom of this file, which times the candidate shapes on the
// caller's batch.  Per system a blocked right-looking LU runs on the CTA's private scratch slice
// (<= 256 x 256, L2 resident) with the current panel and the block row of U in shared memory.  Rows are
// never moved: a permutation maps factor rows to storage rows, so a pivot interchange swaps two integers
// (the factors and the reference's interchange order are the same as with physical swaps).  The solve is
// blocked by 32 rows: one warp per right-hand side substitutes a diagonal block with shuffles, then the
// group folds it into the remaining rows.
//
// It factors in FP32 and refines in FP64: r = b - A x from the caller's FP64 A, d from the FP32
// factors, x += d, until the normwise backward error max_q ||r_q|| / (||A|| ||x_q|| + ||b_q||) is
// <= n 2^-53; a stall or an FP32 pivot <= 10/FLT_MAX refactors that system in FP64.
#include <algorithm>
#include <cfloat>
#include <chrono>
#include <climits>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "panel.cuh"

namespace b2m {
namespace {

constexpr int kBThreads = 256;
constexpr int kBMaxN = 256;
constexpr int kBMaxK = 8;
constexpr int kStrip = 2;  // 16 x 8 tiles per warp step of the trailing update

struct BatchArgs {
    int count;
    const int32_t* n;
    const int32_t* k;
    const int64_t* a_off;
    const int64_t* b_off;
    const double* A;
    const double* B;
    double* X;
    double* scratch;  // the CTAs' factors
    int64_t scratch_cta;  // doubles per CTA (mode 0)
    const int32_t* order;
    int32_t* counter;
    int32_t* info;
    int32_t* iters;
    int mode;
    int small_n;
    int group_warps;
    int big_warps;
    int pw_large, pw_small;
    int max_iter;
};

// a group of threads working on one system, with its own named barrier
struct Grp {
    int tid, nt, bar;
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "r"(nt) : "memory"); }
};

// shared-memory slice of one group
struct Slice {
    double* pan;   // [nmax][pw + 1] panel (factor rows c0.., panel columns)
    double* u;     // [pw][nmax + 1] block row of U right of the panel
    double* y;     // [nmax][kBMaxK] right-hand sides / solution in factor order
    double* red;   // [8] reduction values
    int* redi;     // [8] reduction indices
    int* perm;     // [nmax] storage row of factor row i
    int* flag;     // [4]
    int us;        // row stride of u
    int pw;        // panel width
};

__host__ __device__ inline size_t slice_doubles(int nmax, int pw) {
    return (size_t)nmax * (pw + 1) + (size_t)pw * (nmax + 1) + (size_t)nmax * kBMaxK + 8 + (nmax + 8 + 4 + 1) / 2 + 1;
}

__device__ Slice carve(double* base, int nmax, int pw) {
    Slice s;
    s.pan = base;
    s.u = s.pan + (size_t)nmax * (pw + 1);
    s.y = s.u + (size_t)pw * (nmax + 1);
    s.red = s.y + (size_t)nmax * kBMaxK;
    s.redi = reinterpret_cast<int*>(s.red + 8);
    s.perm = s.redi + 8;
    s.flag = s.perm + nmax;
    s.us = nmax + 1;
    s.pw = pw;
    return s;
}

// factor scratch of one CTA: a matrix of the slice's order per group
__host__ __device__ inline size_t batch_scratch_doubles(int small_n, int G, int GB) {
    const size_t big = (size_t)((kBThreads / 32) / GB) * kBMaxN * kBMaxN;
    const size_t small = (size_t)((kBThreads / 32) / G) * small_n * small_n;
    return big > small ? big : small;
}

template <typename T> __device__ __forceinline__ T sing_thresh();
template <> __device__ __forceinline__ double sing_thresh<double>() { return 10.0 / DBL_MAX; }
template <> __device__ __forceinline__ float sing_thresh<float>() { return 10.0f / FLT_MAX; }

// argmax of |v| over the group (first maximum wins: lowest index among equals); all threads get it
__device__ __forceinline__ void grp_argmax(const Grp& g, const Slice& s, double v, int i, double& bv, int& bi) {
    const int lane = g.tid & 31, w = g.tid >> 5, nw = g.nt >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double v2 = __shfl_xor_sync(0xffffffffu, v, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
        if (i2 >= 0 && (i < 0 || v2 > v || (v2 == v && i2 < i))) { v = v2; i = i2; }
    }
    if (nw == 1) {
        bv = v;
        bi = i;
        return;
    }
    if (lane == 0) { s.red[w] = v; s.redi[w] = i; }
    g.sync();
    bv = -1.0;
    bi = -1;
    for (int q = 0; q < nw; ++q) {
        const double v2 = s.red[q];
        const int i2 = s.redi[q];
        if (i2 >= 0 && (bi < 0 || v2 > bv || (v2 == bv && i2 < bi))) { bv = v2; bi = i2; }
    }
    g.sync();
}

// pivot search over the group: the largest candidate magnitude v >= 0, the lowest row index among
// equal magnitudes (the first maximum of the reference's scan).  A thread without a candidate
// passes v = 0 and i = INT_MAX.  Non-negative doubles order like their bit patterns, so the
// comparison runs on the 64-bit key as two 32-bit warp reductions, then a minimum over the
// indices of the lanes that hold the maximum; the warps' winners are combined the same way.
__device__ __forceinline__ void warp_pivot(double v, int i, double& bv, int& bi) {
    const unsigned long long key = (unsigned long long)__double_as_longlong(v);
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const unsigned mi = __reduce_min_sync(0xffffffffu, (hi == mhi && lo == mlo) ? (unsigned)i : 0xffffffffu);
    bv = __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
    bi = (int)mi;
}

__device__ __forceinline__ void grp_pivot(const Grp& g, const Slice& s, double v, int i, double& bv, int& bi) {
    const int lane = g.tid & 31, w = g.tid >> 5, nw = g.nt >> 5;
    warp_pivot(v, i, bv, bi);
    if (nw == 1) return;
    if (lane == 0) { s.red[w] = bv; s.redi[w] = bi; }
    g.sync();
    warp_pivot(lane < nw ? s.red[lane] : 0.0, lane < nw ? s.redi[lane] : INT_MAX, bv, bi);
    g.sync();
}

// Blocked LU of the n x n matrix A0 (FP64, row-major, ld n) into W (element type T, same layout)
// with row permutation perm.  The first panel reads A0 directly and its updates write every entry
// of W, so A0 is never copied separately.  Global loads are issued in groups before they are used
// (a loop that loads, computes and stores one element at a time pays one L2 latency per element).
// Returns 0, or 1 when a pivot is <= the singular threshold (uniform across the group).
template <typename T>
__device__ int grp_lu(const Grp& g, const Slice& s, const double* A0, T* W, int n, int PW) {
    for (int i = g.tid; i < n; i += g.nt) s.perm[i] = i;
    g.sync();
    const int pwp = PW + 1;
    for (int c0 = 0; c0 < n; c0 += PW) {
        const bool first = c0 == 0;
        auto at = [&](int row, int col) -> T {
            return first ? (T)A0[(int64_t)row * n + col] : W[(int64_t)row * n + col];
        };
        const int pw = min(PW, n - c0), m = n - c0;
        // panel: one factor row per thread, all of its loads in flight
        for (int r = g.tid; r < m; r += g.nt) {
            const int row = s.perm[c0 + r];
            for (int cb = 0; cb < pw; cb += 8) {
                T v[8];
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (cb + c < pw) v[c] = at(row, c0 + cb + c);
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (cb + c < pw) s.pan[r * pwp + cb + c] = (double)v[c];
            }
        }
        g.sync();
        for (int j = 0; j < pw; ++j) {
            double v = -1.0;
            int vi = INT_MAX;
            for (int r = j + g.tid; r < m; r += g.nt) {
                const double a = fabs(s.pan[r * pwp + j]);
                if (a > v) { v = a; vi = r; }  // a NaN never wins
            }
            if (vi == INT_MAX) v = 0.0;
            double bv;
            int pr;
            grp_pivot(g, s, v, vi, bv, pr);
            if (!(bv > (double)sing_thresh<T>())) return 1;
            if (pr != j) {
                for (int c = g.tid; c < pw; c += g.nt) {
                    const double t0 = s.pan[j * pwp + c];
                    s.pan[j * pwp + c] = s.pan[pr * pwp + c];
                    s.pan[pr * pwp + c] = t0;
                }
                if (g.tid == 0) {
                    const int t1 = s.perm[c0 + j];
                    s.perm[c0 + j] = s.perm[c0 + pr];
                    s.perm[c0 + pr] = t1;
                }
            }
            g.sync();
            // reference scaling: the column is multiplied by 1/pivot, in the element type
            const T rinv = (T)1 / (T)s.pan[j * pwp + j];
            for (int r = j + 1 + g.tid; r < m; r += g.nt) {
                const T l = (T)s.pan[r * pwp + j] * rinv;
                s.pan[r * pwp + j] = (double)l;
                for (int c = j + 1; c < pw; ++c)
                    s.pan[r * pwp + c] = (double)((T)s.pan[r * pwp + c] - l * (T)s.pan[j * pwp + c]);
            }
            g.sync();
        }
        for (int r = g.tid; r < m; r += g.nt) {
            T* dst = W + (int64_t)s.perm[c0 + r] * n + c0;
            for (int c = 0; c < pw; ++c) dst[c] = (T)s.pan[r * pwp + c];
        }
        const int c1 = c0 + pw, nr = n - c1;
        if (nr > 0) {
            // block row of U: u = L11^-1 A12 (thread per column, loads in groups of 8)
            for (int c = g.tid; c < nr; c += g.nt) {
                for (int r0 = 0; r0 < pw; r0 += 8) {
                    T v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (r0 + e < pw) v[e] = at(s.perm[c0 + r0 + e], c1 + c);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (r0 + e < pw) s.u[(r0 + e) * s.us + c] = (double)v[e];
                }
                W[(int64_t)s.perm[c0] * n + c1 + c] = (T)s.u[c];
                for (int r = 1; r < pw; ++r) {
                    T acc = (T)s.u[r * s.us + c];
                    for (int q = 0; q < r; ++q) acc -= (T)s.pan[r * pwp + q] * (T)s.u[q * s.us + c];
                    s.u[r * s.us + c] = (double)acc;
                    W[(int64_t)s.perm[c0 + r] * n + c1 + c] = acc;
                }
            }
            g.sync();
            if constexpr (std::is_same<T, double>::value) {
                // trailing update A22 -= L21 U12 on the FP64 tensor cores: warps walk 16 x 8 tiles;
                // m16n8k4 fragments (g = lane / 4, t = lane % 4): a = (L21[g][k+t], L21[g+8][k+t]),
                // b = U12[k+t][g], c = C[g][2t..2t+1], C[g+8][2t..2t+1]
                // A warp takes a 16 x 8 kStrip strip (kStrip 16 x 8 tiles sharing the L21
                // fragment), so that its 4 kStrip loads of C are in flight together.
                const int lane = g.tid & 31, nw = g.nt >> 5, gq = lane >> 2, tq = lane & 3;
                const int tm = (nr + 15) / 16, tn = (nr + 8 * kStrip - 1) / (8 * kStrip);
                for (int tile = g.tid >> 5; tile < tm * tn; tile += nw) {
                    const int r0 = (tile / tn) * 16, q0 = (tile % tn) * 8 * kStrip;
                    const int ra = r0 + gq, rb = r0 + gq + 8;
                    const bool oka = ra < nr, okb = rb < nr;
                    const int rowa = oka ? s.perm[c1 + ra] : 0, rowb = okb ? s.perm[c1 + rb] : 0;
                    double d[kStrip][4];
#pragma unroll
                    for (int u = 0; u < kStrip; ++u) {
                        const int cc = q0 + 8 * u + 2 * tq;
                        d[u][0] = (oka && cc < nr) ? (double)at(rowa, c1 + cc) : 0.0;
                        d[u][1] = (oka && cc + 1 < nr) ? (double)at(rowa, c1 + cc + 1) : 0.0;
                        d[u][2] = (okb && cc < nr) ? (double)at(rowb, c1 + cc) : 0.0;
                        d[u][3] = (okb && cc + 1 < nr) ? (double)at(rowb, c1 + cc + 1) : 0.0;
                    }
                    const double* la = s.pan + (pw + min(ra, nr - 1)) * pwp;
                    const double* lb = s.pan + (pw + min(rb, nr - 1)) * pwp;
                    for (int k = 0; k < pw; k += 4) {
                        const int kk = k + tq;
                        const double a0 = kk < pw ? -la[kk] : 0.0;
                        const double a1 = kk < pw ? -lb[kk] : 0.0;
#pragma unroll
                        for (int u = 0; u < kStrip; ++u) {
                            const int cb = min(q0 + 8 * u + gq, nr - 1);
                            const double b0 = kk < pw ? s.u[kk * s.us + cb] : 0.0;
                            asm volatile(
                                "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
                                "{%0,%1,%2,%3};\n"
                                : "+d"(d[u][0]), "+d"(d[u][1]), "+d"(d[u][2]), "+d"(d[u][3])
                                : "d"(a0), "d"(a1), "d"(b0));
                        }
                    }
                    const int64_t oa = (int64_t)rowa * n + c1, ob = (int64_t)rowb * n + c1;
#pragma unroll
                    for (int u = 0; u < kStrip; ++u) {
                        const int cc = q0 + 8 * u + 2 * tq;
                        if (oka && cc < nr) W[oa + cc] = (T)d[u][0];
                        if (oka && cc + 1 < nr) W[oa + cc + 1] = (T)d[u][1];
                        if (okb && cc < nr) W[ob + cc] = (T)d[u][2];
                        if (okb && cc + 1 < nr) W[ob + cc + 1] = (T)d[u][3];
                    }
                }
            } else {
            // trailing update A22 -= L21 U12: thread per column, 8 rows per step, loads first
            for (int c = g.tid; c < nr; c += g.nt) {
                for (int r0 = 0; r0 < nr; r0 += 8) {
                    T v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = r0 + e < nr ? at(s.perm[c1 + r0 + e], c1 + c) : (T)0;
                    for (int q = 0; q < pw; ++q) {
                        const T uq = (T)s.u[q * s.us + c];
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] -= (T)s.pan[min(pw + r0 + e, m - 1) * pwp + q] * uq;
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (r0 + e < nr) W[(int64_t)s.perm[c1 + r0 + e] * n + c1 + c] = v[e];
                }
            }
            }
            g.sync();
        }
    }
    return 0;
}

// y (factor order, kk columns) <- U^-1 L^-1 y with the factors in W (element type T).  Each
// 32-row diagonal block is staged in shared memory (over the then idle panel / U buffers); one warp
// per right-hand side substitutes it with shuffles, then the group folds it into the other rows.
template <typename T>
__device__ void grp_solve(const Grp& g, const Slice& s, const T* W, int n, int kk) {
    const int lane = g.tid & 31, w = g.tid >> 5, nw = g.nt >> 5;
    const int nb = (n + 31) / 32;
    double* blk = s.pan;  // [32][33], spans into the U buffer for narrow panels
    for (int pass = 0; pass < 2; ++pass) {
        const bool lower = pass == 0;
        for (int bi = 0; bi < nb; ++bi) {
            const int b = lower ? bi : nb - 1 - bi;
            const int b0 = 32 * b, bs = min(32, n - b0);
            for (int base = g.tid; base < 32 * 32; base += 4 * g.nt) {  // four loads in flight
                double v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int e = base + u * g.nt, r = e >> 5, j = e & 31;
                    v[u] = (e < 32 * 32 && r < bs && j < bs) ? (double)W[(int64_t)s.perm[b0 + r] * n + b0 + j] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int e = base + u * g.nt;
                    if (e < 32 * 32) blk[(e >> 5) * 33 + (e & 31)] = v[u];
                }
            }
            g.sync();
            for (int q = w; q < kk; q += nw) {
                const int row = b0 + lane;
                const double* tr = blk + lane * 33;
                double yv = lane < bs ? s.y[row * kBMaxK + q] : 0.0;
                if (lower) {
                    for (int j = 0; j < bs; ++j) {
                        const double xj = __shfl_sync(0xffffffffu, yv, j);
                        if (lane > j) yv = (double)((T)yv - (T)tr[j] * (T)xj);
                    }
                } else {
                    for (int j = bs - 1; j >= 0; --j) {
                        if (lane == j) yv = (double)((T)yv / (T)tr[j]);
                        const double xj = __shfl_sync(0xffffffffu, yv, j);
                        if (lane < j) yv = (double)((T)yv - (T)tr[j] * (T)xj);
                    }
                }
                if (lane < bs) s.y[row * kBMaxK + q] = yv;
            }
            g.sync();
            // fold the block into the other rows: a thread per row, every right-hand side (the
            // row of the factor is read once, 8 loads in flight; same order of terms per entry)
            const int rlo = lower ? b0 + bs : 0, rhi = lower ? n : b0;
            for (int r = rlo + g.tid; r < rhi; r += g.nt) {
                const T* lr = W + (int64_t)s.perm[r] * n + b0;
                T acc[kBMaxK];
#pragma unroll
                for (int q = 0; q < kBMaxK; ++q) acc[q] = q < kk ? (T)s.y[r * kBMaxK + q] : (T)0;
#pragma unroll
                for (int j0 = 0; j0 < 32; j0 += 8) {
                    T v[8];
#pragma unroll
                    for (int e2 = 0; e2 < 8; ++e2) v[e2] = j0 + e2 < bs ? lr[j0 + e2] : (T)0;
#pragma unroll
                    for (int e2 = 0; e2 < 8; ++e2) {
                        if (j0 + e2 < bs) {
                            const double* yr = s.y + (b0 + j0 + e2) * kBMaxK;
#pragma unroll
                            for (int q = 0; q < kBMaxK; ++q)
                                if (q < kk) acc[q] -= v[e2] * (T)yr[q];
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < kBMaxK; ++q)
                    if (q < kk) s.y[r * kBMaxK + q] = (double)acc[q];
            }
            g.sync();
        }
    }
}

// plain FP64 solve of one system
__device__ int solve_plain(const Grp& g, const Slice& s, const BatchArgs& a, int sys, double* W) {
    const int n = a.n[sys], kk = a.k[sys];
    const double* A = a.A + a.a_off[sys];
    if (grp_lu<double>(g, s, A, W, n, s.pw)) return 1;
    const double* B = a.B + a.b_off[sys];
    for (int base = g.tid; base < n * kk; base += 4 * g.nt) {  // four loads in flight
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = base + u * g.nt;
            v[u] = e < n * kk ? B[(int64_t)s.perm[e / kk] * kk + e % kk] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = base + u * g.nt;
            if (e < n * kk) s.y[(e / kk) * kBMaxK + e % kk] = v[u];
        }
    }
    g.sync();
    grp_solve<double>(g, s, W, n, kk);
    double* X = a.X + a.b_off[sys];
    for (int e = g.tid; e < n * kk; e += g.nt) {
        const int i = e / kk, q = e - i * kk;
        X[e] = s.y[i * kBMaxK + q];
    }
    g.sync();
    return 0;
}

// FP32 factorisation + FP64 refinement; returns refinement steps, or -1 when FP64 is needed
__device__ int solve_mixed(const Grp& g, const Slice& s, const BatchArgs& a, int sys, double* Wd) {
    const int n = a.n[sys], kk = a.k[sys];
    float* W = reinterpret_cast<float*>(Wd);
    const double* A = a.A + a.a_off[sys];
    const double* B = a.B + a.b_off[sys];
    double* X = a.X + a.b_off[sys];
    if (grp_lu<float>(g, s, A, W, n, s.pw)) return -1;
    // ||A||inf: a warp per row
    const int lane = g.tid & 31, wp = g.tid >> 5, nw = g.nt >> 5;
    double an = 0.0;
    for (int i = wp; i < n; i += nw) {
        double rs = 0.0;
        for (int j = lane; j < n; j += 32) rs += fabs(A[(int64_t)i * n + j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
        an = fmax(an, rs);
    }
    double bv;
    int bi;
    grp_argmax(g, s, an, 0, bv, bi);
    const double normA = bv;
    for (int e = g.tid; e < n * kk; e += g.nt) X[e] = 0.0;
    // r = b in factor order
    for (int e = g.tid; e < n * kk; e += g.nt) {
        const int i = e / kk, q = e - i * kk;
        s.y[i * kBMaxK + q] = B[(int64_t)s.perm[i] * kk + q];
    }
    g.sync();
    const double tol = (double)n * 0x1.0p-53;
    const int nmax = s.us - 1;
    double* res = s.pan;  // [n][kBMaxK] residual, natural order (the panel buffer is free now)
    unsigned long long* mx = reinterpret_cast<unsigned long long*>(s.pan + (size_t)nmax * kBMaxK);  // [3][8]
    double prev = INFINITY;
    for (int it = 1; it <= a.max_iter; ++it) {
        grp_solve<float>(g, s, W, n, kk);
        for (int e = g.tid; e < n * kk; e += g.nt) {
            const int i = e / kk, q = e - i * kk;
            const double xv = X[e] + s.y[i * kBMaxK + q];
            X[e] = xv;
            s.y[i * kBMaxK + q] = xv;  // x in natural order for the residual below
        }
        if (g.tid < 3 * kBMaxK) mx[g.tid] = 0ull;
        g.sync();
        // r = b - A x in FP64, a warp per row (coalesced rows of A), with the column maxima
        for (int i = wp; i < n; i += nw) {
            double acc[kBMaxK];
#pragma unroll
            for (int q = 0; q < kBMaxK; ++q) acc[q] = 0.0;
            for (int j = lane; j < n; j += 32) {
                const double aij = A[(int64_t)i * n + j];
#pragma unroll
                for (int q = 0; q < kBMaxK; ++q)
                    if (q < kk) acc[q] = fma(aij, s.y[j * kBMaxK + q], acc[q]);
            }
#pragma unroll
            for (int q = 0; q < kBMaxK; ++q) {
                double v = acc[q];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == q && q < kk) {
                    const double bq = B[(int64_t)i * kk + q], xq = s.y[i * kBMaxK + q];
                    const double rq = bq - v;
                    res[i * kBMaxK + q] = rq;
                    atomicMax(&mx[q], (unsigned long long)__double_as_longlong(fabs(rq)));
                    atomicMax(&mx[kBMaxK + q], (unsigned long long)__double_as_longlong(fabs(xq)));
                    atomicMax(&mx[2 * kBMaxK + q], (unsigned long long)__double_as_longlong(fabs(bq)));
                }
            }
        }
        g.sync();
        double eta = 0.0;
        for (int q = 0; q < kk; ++q) {
            const double r1 = __longlong_as_double((long long)mx[q]);
            const double x1 = __longlong_as_double((long long)mx[kBMaxK + q]);
            const double b1 = __longlong_as_double((long long)mx[2 * kBMaxK + q]);
            const double den = normA * x1 + b1;
            eta = fmax(eta, den > 0.0 ? r1 / den : (r1 > 0.0 ? INFINITY : 0.0));
        }
        for (int e = g.tid; e < n * kk; e += g.nt) {
            const int i = e / kk, q = e - i * kk;
            s.y[i * kBMaxK + q] = res[s.perm[i] * kBMaxK + q];
        }
        g.sync();
        if (eta <= tol) return it;
        if (!(eta < INFINITY) || (it >= 2 && eta > 0.5 * prev)) return -1;
        prev = eta;
    }
    return -1;
}

// FP32 factor + FP64 refinement (mode 1).  At most 128 registers a thread, so that
// two CTAs share an SM whenever the tile shape's shared memory allows it.
__global__ void __launch_bounds__(kBThreads, 2) batch_solve_kernel(BatchArgs a) {
    extern __shared__ __align__(16) double bsm[];
    __shared__ int s_sys[8];
    const int t = threadIdx.x;
    double* W = a.scratch + (size_t)blockIdx.x * batch_scratch_doubles(a.small_n, a.group_warps, a.big_warps);
    for (;;) {
        if (t == 0) s_sys[0] = atomicAdd(a.counter, 1);
        __syncthreads();
        const int idx = s_sys[0];
        __syncthreads();
        if (idx >= a.count) return;
        // this system and up to ng - 1 more from the queue, one per group; the first one decides
        // the round's group size and slice shape (the queue is sorted largest first, so a round
        // that starts with a large system may end with small ones, which fit its slices too)
        const bool big = a.n[a.order[idx]] > a.small_n;
        const int gw = big ? a.big_warps : a.group_warps, ng = (kBThreads / 32) / gw;
        const int nmax = big ? kBMaxN : a.small_n, pw = big ? a.pw_large : a.pw_small;
        if (t == 0) {
            for (int q = 1; q < ng; ++q) {
                const int j = atomicAdd(a.counter, 1);
                s_sys[q] = j < a.count ? j : -1;
            }
        }
        __syncthreads();
        const int gi = t / (32 * gw);
        const int myidx = s_sys[gi];
        if (myidx >= 0) {
            const int msys = a.order[myidx];
            const Grp g{t - gi * 32 * gw, 32 * gw, 2 + gi};
            const Slice s = carve(bsm + (size_t)gi * slice_doubles(nmax, pw), nmax, pw);
            double* Wg = W + (size_t)gi * nmax * nmax;
            const int iters = solve_mixed(g, s, a, msys, Wg);
            const int st = iters < 0 ? solve_plain(g, s, a, msys, Wg) : 0;
            if (g.tid == 0) {
                a.info[msys] = st;
                if (a.iters) a.iters[msys] = iters;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// FP64 systems (mode 0): one launch of persistent CTAs of four warps, three to an SM.  A CTA takes one
// system of order > 128 on all four warps, two of order 65 .. 128 on two warps each, or four smaller
// ones on a warp each.  What bounds a system is the chain of its columns (pivot search, reciprocal,
// update of the next column), so the chain is kept short and several systems share an SM to fill it:
//   * leaves of 32 (16 for two warps or one) columns, their rows in shared memory and, eight columns
//     at a time, in registers that shift left by one per column (a compact loop; see panel.cu, whose
//     elimination this is for one CTA): one barrier a column;
//   * rows never move: a thread carries its rows' positions, a permutation maps positions to rows;
//   * the right-hand sides are extra columns, so L is never stored and needs no forward sweep;
//   * U12 and the trailing update with it run on the FP64 tensor cores, a strip of columns per warp
//     from registers (lu_strip);
//   * the back substitution multiplies by the diagonal's reciprocal and corrects by the exact residual
//     (as accurate as the division, whose 144 cycles would be on its chain 256 times), one warp per
//     block with four lanes a right-hand side, and folds blocks on the tensor cores.
// The matrix is worked on in the CTA's scratch (L2); the first leaf and update read A itself.
// Measured on a B200: 20,000 systems of order 8 .. 256, k 1 .. 4: 23.0 ms before (panel and update of a
// system on 8 warps, the panel in shared memory) and 8.8 ms (6.5 TFLOP/s) now; one system alone of order
// 100 94 us, 256 326 us.
// ------------------------------------------------------------------------------------------
constexpr int kLuThreads = 128;
constexpr int kLuCtas = 3;           // CTAs per SM the registers and the shared memory allow
constexpr int kBk = 8;               // columns per register block

struct __align__(16) LuCand {
    double rinv;      // 1 / row[0]
    int pos, lrow;    // position below the leaf's top, row in S
    double row[kBk];  // the row's block columns, from the current one on
};

// shared memory of one group
template <int NW, int W> struct LuSlice {
    static constexpr int kRows = NW * 64;
    double S[kRows * W];         // the leaf's rows, 16-byte pairs swizzled by row
    double u[W * W];             // U11; then L11^T
    double l8[kBk * kBk];        // a block's L
    LuCand cand[2][NW];
    __align__(16) uint32_t key[2][4];  // leading words of the candidates
    int pl[W];                   // pivot rows in S
    uint16_t perm[kRows];        // position -> row of the matrix
    uint16_t lrow[kRows];        // live position -> row in S
};

template <int NW> __device__ __forceinline__ void lu_sync(int bar) {
    if constexpr (NW == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "n"(NW * 32) : "memory");
}

// Leaf of w <= W columns over m rows (loaded in s.S, zero past column w): eliminates with partial
// pivoting.  pos[r] of row t + r * NW * 32 (its position on entry): its position afterwards, or
// -1 - j for the pivot of column j.  Multipliers are left in S, U11 in s.u; ipiv (may be null): ipiv[j] = c0 + the
// position column j's pivot row had.  False: singular.
template <int NW, int W>
__device__ __forceinline__ bool lu_leaf(LuSlice<NW, W>& s, int t, int bar, int w, int m, int (&pos)[2],
                                        int32_t* ipiv = nullptr, int c0 = 0) {
    constexpr int NT = NW * 32, RPT = 2;
    const int lane = t & 31, warp = t >> 5;
    double* S = s.S;
    auto sx = [](int row, int c) { return row * W + 2 * ((c >> 1) ^ (row & 7)) + (c & 1); };
    double act[RPT][kBk];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int i = 0; i < kBk; i += 2) {
            const double2 x = pos[r] >= 0 ? *reinterpret_cast<const double2*>(S + sx(t + r * NT, i))
                                          : make_double2(0.0, 0.0);
            act[r][i] = x.x; act[r][i + 1] = x.y;
        }
    auto publish = [&](const int col) {
        uint32_t h[RPT];
#pragma unroll
        for (int r = 0; r < RPT; ++r) h[r] = pos[r] >= 0 ? mag_hi(act[r][0]) : 0u;
        const uint32_t mh = max(h[0], h[1]);
        const bool second = h[1] > h[0];
        double cr[kBk];
#pragma unroll
        for (int i = 0; i < kBk; ++i) cr[i] = second ? act[1][i] : act[0][i];
        int cp = second ? pos[1] : pos[0], cl = second ? t + NT : t;
        cr[0] = mh != 0 ? cr[0] : 0.0;
        double rarg;  // opaque: a lane without a candidate must not divide by its zero (slow path)
        asm("{ .reg .pred p; setp.ne.u32 p, %2, 0; selp.f64 %0, %1, 0d3FF0000000000000, p; }"
            : "=d"(rarg)
            : "d"(cr[0]), "r"(mh));
        double rinv = 1.0 / rarg;
        const uint32_t M = __reduce_max_sync(0xffffffffu, mh);
        const uint32_t b1 = __ballot_sync(0xffffffffu, mh == M);
        const uint32_t b2 = __ballot_sync(0xffffffffu, mh == M && h[0] == h[1]);
        int wl = __ffs(b1) - 1;
        if (M != 0 && ((b1 & (b1 - 1)) || b2 || M >= kInfHi)) {
            double ba = 0.0;
            cp = 0x7fffffff;
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const double a = fabs(act[r][0]);
                if (pos[r] >= 0 && a > 0.0 && (a > ba || (a == ba && pos[r] < cp))) {
                    ba = a;
                    cp = pos[r];
                    cl = t + r * NT;
#pragma unroll
                    for (int i = 0; i < kBk; ++i) cr[i] = act[r][i];
                }
            }
            if (!(ba > 0.0)) cr[0] = 0.0;
            rinv = 1.0 / (ba > 0.0 ? cr[0] : 1.0);
            wl = warp_winner(ba, cp);
        }
        if (lane == wl) {
            LuCand& c = s.cand[col & 1][warp];
#pragma unroll
            for (int i = 0; i < kBk; i += 2)
                *reinterpret_cast<double2*>(&c.row[i]) = make_double2(cr[i], cr[i + 1]);
            c.rinv = rinv;
            *reinterpret_cast<int2*>(&c.pos) = make_int2(M != 0 ? cp : 0x7fffffff, cl);
            s.key[col & 1][warp] = mag_hi(cr[0]);
        }
    };
    publish(0);
    for (int jb = 0; jb < w; jb += kBk) {
        const int bw = min(kBk, w - jb);
#pragma unroll 1
        for (int q = 0; q < bw; ++q) {
            const int j = jb + q;
            lu_sync<NW>(bar);
            int win = 0;
            if constexpr (NW > 1) {
                const uint4 kv = *reinterpret_cast<const uint4*>(&s.key[j & 1][0]);
                const uint32_t k[4] = {kv.x, kv.y, kv.z, kv.w};
                uint32_t M = k[0];
                int n = 0;
#pragma unroll
                for (int e = 1; e < NW; ++e) M = max(M, k[e]);
#pragma unroll
                for (int e = NW - 1; e >= 0; --e) {
                    win = k[e] == M ? e : win;
                    n += k[e] == M ? 1 : 0;
                }
                if (n > 1) {
                    win = warp_winner(lane < NW ? fabs(s.cand[j & 1][lane].row[0]) : 0.0,
                                    lane < NW ? s.cand[j & 1][lane].pos : 0x7fffffff);
                    if (win >= NW) win = 0;
                }
            }
            const LuCand& b = s.cand[j & 1][win];
            double u[kBk];
#pragma unroll
            for (int i = 0; i < kBk; i += 2) {
                const double2 x = *reinterpret_cast<const double2*>(&b.row[i]);
                u[i] = x.x; u[i + 1] = x.y;
            }
            const double rinv = b.rinv;
            const int2 pl = *reinterpret_cast<const int2*>(&b.pos);
            if (!(fabs(u[0]) > sing_thresh<double>())) return false;  // uniform: every warp read the same
            if (warp == NW - 1) {  // the pivot row's part of U inside its block
                if (lane < kBk && q + lane < kBk && j + lane < W) s.u[j * W + j + lane] = b.row[lane];
                if (lane == 0) {
                    s.pl[j] = pl.y;
                    if (ipiv) ipiv[j] = c0 + pl.x;
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int rl = t + r * NT;
                if (rl == pl.y) pos[r] = -1 - j;
                else if (pos[r] == j) pos[r] = pl.x;
                const double l = act[r][0] * rinv + 0.0;
                if (pos[r] >= 0) S[sx(rl, j)] = l;
#pragma unroll
                for (int i = 1; i < kBk; ++i) act[r][i - 1] = fma(-l, u[i], act[r][i]);
                act[r][kBk - 1] = 0.0;
            }
            if (q + 1 < bw) publish(j + 1);
        }
        const int c1 = jb + kBk;
        if (c1 >= w) break;
        // block end: the pivot rows right of the block, solved with the block's L
        lu_sync<NW>(bar);
        for (int e = t; e < kBk * (W / 2); e += NT) {
            const int q = e / (W / 2), c = 2 * (e - q * (W / 2));
            const double2 x = *reinterpret_cast<const double2*>(S + sx(s.pl[jb + q], c));
            if (c >= c1) *reinterpret_cast<double2*>(&s.u[(jb + q) * W + c]) = x;
            else if (c >= jb) *reinterpret_cast<double2*>(&s.l8[q * kBk + c - jb]) = x;
        }
        lu_sync<NW>(bar);
        if (warp == 0 && c1 + lane < W) {
            const int c = c1 + lane;
            double x[kBk];
#pragma unroll
            for (int q = 0; q < kBk; ++q) x[q] = s.u[(jb + q) * W + c];
#pragma unroll
            for (int q0 = 0; q0 < kBk - 1; ++q0)
#pragma unroll
                for (int q1 = q0 + 1; q1 < kBk; ++q1) x[q1] = fma(-s.l8[q1 * kBk + q0], x[q0], x[q1]);
#pragma unroll
            for (int q = 1; q < kBk; ++q) s.u[(jb + q) * W + c] = x[q];
        }
        double l[RPT][kBk];
#pragma unroll
        for (int r = 0; r < RPT; ++r)
#pragma unroll
            for (int q = 0; q < kBk; q += 2) {
                double2 x = make_double2(0.0, 0.0), y = x;
                if (pos[r] >= 0) {
                    x = *reinterpret_cast<const double2*>(S + sx(t + r * NT, jb + q));
                    y = *reinterpret_cast<const double2*>(S + sx(t + r * NT, c1 + q));
                }
                l[r][q] = x.x; l[r][q + 1] = x.y;
                act[r][q] = y.x; act[r][q + 1] = y.y;
            }
        lu_sync<NW>(bar);
#pragma unroll
        for (int i = 0; i < kBk; i += 2)
#pragma unroll
            for (int q = 0; q < kBk; ++q) {
                const double2 uu = *reinterpret_cast<const double2*>(&s.u[(jb + q) * W + c1 + i]);
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    act[r][i] = fma(-l[r][q], uu.x, act[r][i]);
                    act[r][i + 1] = fma(-l[r][q], uu.y, act[r][i + 1]);
                }
            }
        publish(c1);
#pragma unroll 1
        for (int c = c1 + kBk; c < w; c += 2) {
            double2 x[RPT];
#pragma unroll
            for (int r = 0; r < RPT; ++r)
                x[r] = pos[r] >= 0 ? *reinterpret_cast<const double2*>(S + sx(t + r * NT, c)) : make_double2(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < kBk; ++q) {
                const double2 uu = *reinterpret_cast<const double2*>(&s.u[(jb + q) * W + c]);
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    x[r].x = fma(-l[r][q], uu.x, x[r].x);
                    x[r].y = fma(-l[r][q], uu.y, x[r].y);
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r)
                if (pos[r] >= 0) *reinterpret_cast<double2*>(S + sx(t + r * NT, c)) = x[r];
        }
    }
    return true;
}

__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a0), "d"(a1), "d"(b));
}

// A strip of 16 columns from q0 on, right of the leaf [c0, c0 + w): U12 = L11^-1 A12 in registers,
// then the strip's part of the trailing update with it, on the FP64 tensor cores (m16n8k4).
//
// Lane (g, t) = (lane / 4, lane % 4) holds of every 8 rows of A12 rows 2 t and 2 t + 1, columns g and
// g + 8 of each 16: the accumulator layout of X^T (16 columns x 8 rows), which is also the operand
// layout of X^T for the blocks below and of U12 for the trailing update when the k index of step s
// (0, 1) counts rows 2 t + s.  So neither shared memory nor shuffles lie between the solve and the
// updates; only the 8 x 8 triangles go by substitution, with a shuffle per row.  (A thread per column
// read each multiplier by a broadcast, which costs the SM's shared memory 2 cycles per warp: 10,600
// cycles a leaf of order 256.)  kSum: the trailing update's products are summed before they meet the old value
// (as in the products of the larger orders' factorisation; a third of the rounding, but registers that three CTAs
// an SM do not have).
template <int NW, int W, bool kFirst, bool kSum = false>
__device__ __forceinline__ void lu_strip(LuSlice<NW, W>& s, int lane, const double* A, int64_t lda, const double* B,
                                         int n, int kk, int ld, double* V, int c0, int w, int q0) {
    const int g = lane >> 2, t = lane & 3, nt = n + kk, cb = c0 + w, mr = n - cb;
    auto sx = [](int row, int c) { return row * W + 2 * ((c >> 1) ^ (row & 7)) + (c & 1); };
    // Element (row, col) as this step finds it: A and B before the first update (kFirst).  Columns past
    // the last one read it again, so that no load hides behind a branch; they are not stored.
    auto at = [&](int row, int col) {
        const int c = min(col, nt - 1);
        if constexpr (kFirst) return c < n ? A[row * lda + c] : B[row * kk + c - n];
        else return V[row * ld + c];
    };
    double x[W / 8][4];
#pragma unroll
    for (int b = 0; b < W / 8; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int row = s.perm[c0 + min(8 * b + 2 * t + e, w - 1)];
#pragma unroll
            for (int h = 0; h < 2; ++h) x[b][2 * h + e] = at(row, q0 + 8 * h + g);
        }
    // Rows past w (the last leaf of a matrix) hold copies of its last row: nothing depends on them and
    // they are not stored.
#pragma unroll
    for (int b = 0; b < W / 8; ++b) {
        const int pa = s.pl[min(8 * b + 2 * t, w - 1)], pb = s.pl[min(8 * b + 2 * t + 1, w - 1)];
        double2 la[4], lb[4];  // this lane's two rows of the triangle
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            la[r] = *reinterpret_cast<const double2*>(s.S + sx(pa, 8 * b + 2 * r));
            lb[r] = *reinterpret_cast<const double2*>(s.S + sx(pb, 8 * b + 2 * r));
        }
#pragma unroll
        for (int r = 0; r < 7; ++r) {
            const double ma = r & 1 ? la[r / 2].y : la[r / 2].x, mb = r & 1 ? lb[r / 2].y : lb[r / 2].x;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double v = __shfl_sync(0xffffffffu, x[b][2 * h + (r & 1)], (lane & ~3) + r / 2);
                if (2 * t > r) x[b][2 * h] = fma(-ma, v, x[b][2 * h]);
                if (2 * t + 1 > r) x[b][2 * h + 1] = fma(-mb, v, x[b][2 * h + 1]);
            }
        }
#pragma unroll
        for (int b2 = b + 1; b2 < W / 8; ++b2) {
            const double2 l = *reinterpret_cast<const double2*>(s.S + sx(s.pl[min(8 * b2 + g, w - 1)], 8 * b + 2 * t));
            dmma(x[b2], x[b][0], x[b][2], -l.x);
            dmma(x[b2], x[b][1], x[b][3], -l.y);
        }
    }
#pragma unroll
    for (int b = 0; b < W / 8; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = 8 * b + 2 * t + e;
            double* dst = V + s.perm[c0 + min(j, w - 1)] * ld + q0 + g;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (j < w && q0 + g + 8 * h < nt) dst[8 * h] = x[b][2 * h + e];
                x[b][2 * h + e] = -x[b][2 * h + e];
            }
        }
    if (mr <= 0) return;
    // Rows below (w = W): 16 x 8 tiles, c = rows g, g + 8, columns 2 t, 2 t + 1; the next tile's old
    // values are in flight under this one's products.  Pairs of columns are aligned in V, whose rows
    // have a spare element where their length is odd; tiles past the last row repeat it.
    double old[2][4];
    int ro[2];
    auto fetch = [&](int r0, int (&rows)[2]) {
#pragma unroll
        for (int e = 0; e < 2; ++e) rows[e] = s.perm[cb + min(r0 + g + 8 * e, mr - 1)];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = q0 + 8 * h + 2 * t;
                if constexpr (kFirst) {
                    old[h][2 * e] = at(rows[e], c);
                    old[h][2 * e + 1] = at(rows[e], c + 1);
                } else {
                    const double2 v = *reinterpret_cast<const double2*>(V + rows[e] * ld + min(c, ld - 2));
                    old[h][2 * e] = v.x;
                    old[h][2 * e + 1] = v.y;
                }
            }
    };
    fetch(0, ro);
#pragma unroll 1
    for (int r0 = 0; r0 < mr; r0 += 16) {
        double acc[2][4], add[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[h][e] = kSum ? 0.0 : old[h][e];
                add[h][e] = old[h][e];
            }
        const int la = s.lrow[w + min(r0 + g, mr - 1)], lb = s.lrow[w + min(r0 + g + 8, mr - 1)];
        int rn[2] = {ro[0], ro[1]};
        if (r0 + 16 < mr) fetch(r0 + 16, rn);
#pragma unroll
        for (int b = 0; b < W / 8; ++b) {
            const double2 a0 = *reinterpret_cast<const double2*>(s.S + sx(la, 8 * b + 2 * t));
            const double2 a1 = *reinterpret_cast<const double2*>(s.S + sx(lb, 8 * b + 2 * t));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                dmma(acc[h], a0.x, a1.x, x[b][2 * h]);
                dmma(acc[h], a0.y, a1.y, x[b][2 * h + 1]);
            }
        }
        if constexpr (kSum)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[h][e] += add[h][e];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            double* dst = V + ro[e] * ld + q0 + 2 * t;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (r0 + g + 8 * e < mr && q0 + 8 * h + 2 * t < nt)
                    *reinterpret_cast<double2*>(dst + 8 * h) = make_double2(acc[h][2 * e], acc[h][2 * e + 1]);
        }
        ro[0] = rn[0];
        ro[1] = rn[1];
    }
}

// y <- U^-1 y (y: n x 8 in s.S), U in the rows V[s.perm[i]] (stride ld); a block of U goes to s.u.
template <int NW, int W>
__device__ __forceinline__ void lu_upper(LuSlice<NW, W>& s, int t, int bar, const double* V, int64_t ld, int n) {
    constexpr int NT = NW * 32;
    const int lane = t & 31, warp = t >> 5;
    double* y = s.S;
    for (int b0 = (n - 1) / W * W; b0 >= 0; b0 -= W) {
        const int bs = min(W, n - b0);
        lu_sync<NW>(bar);
        batched_copy<NT, 8, double>(t, W * W,  // the block's columns: u[c][r] = U(b0 + r, b0 + c), identity past bs
            [&](int e) {
                const int r = e / W, c = e % W;
                return (r <= c && c < bs) ? V[s.perm[b0 + r] * ld + b0 + c] : (r == c ? 1.0 : 0.0);
            },
            [&](int e, double v) { s.u[e % W * W + e / W] = v; });
        lu_sync<NW>(bar);
        if (warp == 0) {
            // lane = right-hand side + 8 * (row & 3); rows from the last one up, four a step.  x / d is
            // the product with the reciprocal corrected by its exact residual; where a diagonal is far
            // from 1 the block, and where a result is not finite its right-hand side, is solved with
            // divisions.  So a right-hand side's result does not depend on its neighbours.
            const int q = lane & 7, rg = lane >> 3;
            double dv[W / 4], di[W / 4];
            bool odd = false;
#pragma unroll
            for (int i = 0; i < W / 4; ++i) {
                dv[i] = s.u[(4 * i + rg) * (W + 1)];
                di[i] = 1.0 / dv[i];
                odd = odd || mag_hi(dv[i]) - 0x01700000u >= 0x7d000000u;  // outside 2^-1000 .. 2^1000
            }
            double y0[W / 4];
#pragma unroll
            for (int i = 0; i < W / 4; ++i) y0[i] = 4 * i + rg < bs ? y[(b0 + 4 * i + rg) * kBMaxK + q] : 0.0;
            auto solve = [&](auto divide, bool put) {
                constexpr bool kDivide = decltype(divide)::value;
                constexpr int kTop = W / 4 - 1;
                double x[W / 4], d[W / 4], r[W / 4];
#pragma unroll
                for (int i = 0; i < W / 4; ++i) {
                    x[i] = y0[i];
                    d[i] = dv[i];
                    r[i] = di[i];
                }
                bool finite = true;
#pragma unroll 1
                for (int i4 = kTop; i4 >= 0; --i4) {
#pragma unroll
                    for (int v = 3; v >= 0; --v) {
                        const double z = x[kTop];
                        double xq;
                        if constexpr (kDivide) {
                            xq = z / d[kTop];
                        } else {
                            xq = z * r[kTop];
                            xq = fma(fma(-xq, d[kTop], z), r[kTop], xq);
                        }
                        const double xj = __shfl_sync(0xffffffffu, xq, q + 8 * v);
                        if (rg == v) x[kTop] = xq;
                        const double* uc = &s.u[(4 * i4 + v) * W + rg];
                        if (rg < v) x[kTop] = fma(-uc[4 * i4], xj, x[kTop]);
#pragma unroll
                        for (int i = 1; i < W / 4; ++i)
                            if (i4 - i >= 0) x[kTop - i] = fma(-uc[4 * (i4 - i)], xj, x[kTop - i]);
                    }
                    finite = finite && mag_hi(x[kTop]) < kInfHi;
                    if (put && 4 * i4 + rg < bs) y[(b0 + 4 * i4 + rg) * kBMaxK + q] = x[kTop];
#pragma unroll
                    for (int i = kTop; i > 0; --i) {
                        x[i] = x[i - 1];
                        d[i] = d[i - 1];
                        r[i] = r[i - 1];
                    }
                }
                return finite;
            };
            uint32_t again = __any_sync(0xffffffffu, odd) ? 0xffffffffu : 0u;
            if (!again) again = __ballot_sync(0xffffffffu, !solve(std::false_type{}, true));
            if (again) solve(std::true_type{}, (again & (0x01010101u << q)) != 0);
        }
        lu_sync<NW>(bar);
        // fold the block into the rows above (only full blocks of 4 k: bs < W only in the last one)
        const int g = lane >> 2, tq = lane & 3;
        for (int r0 = 16 * warp; r0 < b0; r0 += 16 * NW) {
            const int64_t ra = s.perm[r0 + g] * ld + b0, rb = s.perm[r0 + g + 8] * ld + b0;  // (b0 is a multiple of 16)
            double a0[W / 4], a1[W / 4], acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < W / 4; ++k) {
                const bool in = 4 * k + tq < bs;
                a0[k] = in ? V[ra + 4 * k + tq] : 0.0;
                a1[k] = in ? V[rb + 4 * k + tq] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < W / 4; ++k) {
                const double b = 4 * k + tq < bs ? y[(b0 + 4 * k + tq) * kBMaxK + g] : 0.0;
                asm volatile(
                    "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                    : "+d"(acc[0]), "+d"(acc[1]), "+d"(acc[2]), "+d"(acc[3])
                    : "d"(a0[k]), "d"(a1[k]), "d"(b));
            }
            double2* ya = reinterpret_cast<double2*>(y + (r0 + g) * kBMaxK + 2 * tq);
            double2* yb = reinterpret_cast<double2*>(y + (r0 + g + 8) * kBMaxK + 2 * tq);
            *ya = make_double2(ya->x - acc[0], ya->y - acc[1]);
            *yb = make_double2(yb->x - acc[2], yb->y - acc[3]);
        }
    }
}

// One system on a group of NW warps; V is its scratch (row stride ld, 16-byte aligned rows).  0, or 1
// when singular (uniform over the group).
template <int NW, int W>
__device__ __forceinline__ int lu_system(LuSlice<NW, W>& s, int t, int bar, const double* A, const double* B, double* X,
                                         int n, int kk, double* V) {
    constexpr int NT = NW * 32;
    const int lane = t & 31, warp = t >> 5, ld = (n + kk + 1) & ~1, nt = n + kk;
    auto sx = [](int row, int c) { return row * W + 2 * ((c >> 1) ^ (row & 7)) + (c & 1); };
    for (int i = t; i < n; i += NT) s.perm[i] = (uint16_t)i;
    lu_sync<NW>(bar);
    for (int c0 = 0; c0 < n; c0 += W) {
        const bool first = c0 == 0;
        const int w = min(W, n - c0), m = n - c0, cb = c0 + w;
        if (first) {
#pragma unroll 4
            for (int e = t; e < m * W; e += NT) {
                const int rl = e / W, c = e % W;
                cp_async8(s.S + sx(rl, c), c < w ? A + (int64_t)rl * n + c : A, c < w ? 8 : 0);
            }
        } else {
#pragma unroll 4
            for (int e = t; e < m * (W / 2); e += NT) {
                const int rl = e / (W / 2), c = 2 * (e % (W / 2));
                cp_async16(s.S + sx(rl, c), c < w ? V + s.perm[c0 + rl] * ld + c0 + c : V,
                           c + 1 < w ? 16 : (c < w ? 8 : 0));
            }
        }
        cp_async_commit();
        int pos[2], row[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int rl = t + r * NT;
            pos[r] = rl < m ? rl : -1 - W;
            row[r] = rl < m ? s.perm[c0 + rl] : 0;
        }
        cp_async_wait<0>();
        lu_sync<NW>(bar);
        if (!lu_leaf<NW, W>(s, t, bar, w, m, pos)) return 1;
        lu_sync<NW>(bar);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int rl = t + r * NT;
            if (rl < m) s.perm[c0 + (pos[r] < 0 ? -1 - pos[r] : pos[r])] = (uint16_t)row[r];
            if (rl < m && pos[r] >= 0) s.lrow[pos[r]] = (uint16_t)rl;
        }
        lu_sync<NW>(bar);
        for (int e0 = t; e0 < W * W; e0 += 4 * NT) {  // U11
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = e0 + i * NT, j = e / W, c = e % W;
                if (j < w && c >= j && c < w) V[s.perm[c0 + j] * ld + c0 + c] = s.u[e];
            }
        }
        // the columns to the right, 16 a warp (strips of 32 took 10.5 ms instead of 8.8: more registers
        // than three CTAs an SM allow, and idle warps on the last columns)
        auto strips = [&](auto first) {
            constexpr bool kFirst = decltype(first)::value;
            for (int q0 = cb + 16 * warp; q0 < nt; q0 += 16 * NW)
                lu_strip<NW, W, kFirst>(s, lane, A, n, B, n, kk, ld, V, c0, w, q0);
        };
        if (first) strips(std::true_type{});
        else strips(std::false_type{});
        lu_sync<NW>(bar);
    }
    // ---- back substitution: y (n x 8, zero past kk) in S's place, a block of U in u
    double* y = s.S;
    for (int e = t; e < n * kBMaxK; e += NT) {
        const int j = e / kBMaxK, q = e % kBMaxK;
        y[e] = q < kk ? V[s.perm[j] * ld + n + q] : 0.0;
    }
    lu_upper<NW, W>(s, t, bar, V, ld, n);
    lu_sync<NW>(bar);
    for (int e = t; e < n * kk; e += NT) X[e] = y[e / kk * kBMaxK + e % kk];
    lu_sync<NW>(bar);
    return 0;
}

// scratch of one system with its right-hand sides; of a CTA in a batch whose largest order is nmax
__host__ __device__ constexpr int64_t lu_mat(int n) { return (int64_t)n * ((n + kBMaxK + 1) & ~1); }
int64_t lu_scratch(int nmax) { return std::max(nmax > 64 ? 2 * lu_mat(128) : 4 * lu_mat(64), lu_mat(nmax)); }

union LuShared {
    LuSlice<4, 32> one;
    LuSlice<2, 16> two[2];
    LuSlice<1, 16> four[4];
};

// As many CTAs as systems: the time of one counts, not how many an SM holds (four warps each against two or
// one: order 100 95 / 115 us, 200 of order 60 60 / 68 us, 440 of order 100 131 / 134 us).
bool lu_wide(int64_t count, int num_sms) { return count <= (int64_t)num_sms * kLuCtas; }

// wide: every system runs on four warps (few systems, where the time of one counts)
__global__ void __launch_bounds__(kLuThreads, kLuCtas) batch_lu_kernel(BatchArgs a, int wide) {
    extern __shared__ __align__(16) unsigned char lu_dyn[];
    LuShared& sh = *reinterpret_cast<LuShared*>(lu_dyn);
    __shared__ int s_sys[4];
    const int t = threadIdx.x;
    double* V = a.scratch + (size_t)blockIdx.x * a.scratch_cta;
    for (;;) {
        if (t == 0) s_sys[0] = atomicAdd(a.counter, 1);
        __syncthreads();
        const int idx = s_sys[0];
        if (idx >= a.count) return;
        // the queue is sorted largest first: the systems that follow are no larger
        const int n0 = a.n[a.order[idx]];
        const int groups = wide || n0 > 128 ? 1 : (n0 > 64 ? 2 : 4);
        if (t > 0 && t < groups) {
            const int j = atomicAdd(a.counter, 1);
            s_sys[t] = j < a.count ? j : -1;
        }
        __syncthreads();
        const int gi = t / (kLuThreads / groups), myidx = s_sys[gi], gt = t - gi * (kLuThreads / groups);
        if (myidx >= 0) {
            const int sys = a.order[myidx], n = a.n[sys], kk = a.k[sys];
            const double *A = a.A + a.a_off[sys], *B = a.B + a.b_off[sys];
            double* X = a.X + a.b_off[sys];
            int st;
            if (groups == 1) st = lu_system<4, 32>(sh.one, gt, 1, A, B, X, n, kk, V);
            else if (groups == 2) st = lu_system<2, 16>(sh.two[gi], gt, 1 + gi, A, B, X, n, kk, V + gi * lu_mat(128));
            else st = lu_system<1, 16>(sh.four[gi], gt, 0, A, B, X, n, kk, V + gi * lu_mat(64));
            if (gt == 0) {
                a.info[sys] = st;
                if (a.iters) a.iters[sys] = 0;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// One system of order <= 256 in the calls on a single matrix: its factorisation in place (small_lu_kernel)
// and the solves with its factors (small_solve_kernel), one launch each, on the parts above.  The recursion of
// the larger orders needs four launches a leaf here (panel, interchanges, U12, update), each shorter than
// the gap to the next; its solve a copy, a gather and two sweeps.
//
// small_lu_kernel: four warps do the leaves, eight the strips.  L is kept too, in its storage row; rows go to
// their positions at the end, from the scratch V (n rows of (n + 1) & ~1) back to A.
// Measured on a B200 (factor and one right-hand side, the whole call): order 100 201 us before and 125 us now,
// order 256 429 and 339 us; the inverse of order 100 230 and 129 us.
// ------------------------------------------------------------------------------------------
constexpr int kSmThreads = 256;

__global__ void __launch_bounds__(kSmThreads, 1)
    small_lu_kernel(double* A, int64_t ld, int n, double* V, int32_t* ipiv, int32_t* perm, int32_t* status) {
    constexpr int W = 32;
    extern __shared__ __align__(16) unsigned char lu_dyn[];
    LuSlice<4, W>& s = *reinterpret_cast<LuSlice<4, W>*>(lu_dyn);
    __shared__ int16_t s_pos[kBMaxN];   // of a leaf's rows: position (-1 - j: the pivot of column j),
    __shared__ uint16_t s_row[kBMaxN];  // storage row
    __shared__ int s_stop;
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, ldv = (n + 1) & ~1;
    auto sx = [](int row, int c) { return row * W + 2 * ((c >> 1) ^ (row & 7)) + (c & 1); };
    for (int i = t; i < n; i += kSmThreads) s.perm[i] = (uint16_t)i;
    if (t == 0) s_stop = 0;
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += W) {
        const bool first = c0 == 0;
        const int w = min(W, n - c0), m = n - c0, cb = c0 + w;
        if (first) {
#pragma unroll 4
            for (int e = t; e < m * W; e += kSmThreads) {
                const int rl = e / W, c = e % W;
                cp_async8(s.S + sx(rl, c), c < w ? A + rl * ld + c : A, c < w ? 8 : 0);
            }
        } else {
#pragma unroll 4
            for (int e = t; e < m * (W / 2); e += kSmThreads) {
                const int rl = e / (W / 2), c = 2 * (e % (W / 2));
                cp_async16(s.S + sx(rl, c), c < w ? V + s.perm[c0 + rl] * ldv + c0 + c : V,
                           c + 1 < w ? 16 : (c < w ? 8 : 0));
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        if (t < 128) {
            int pos[2], row[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int rl = t + r * 128;
                pos[r] = rl < m ? rl : -1 - W;
                row[r] = rl < m ? s.perm[c0 + rl] : 0;
            }
            const bool ok = lu_leaf<4, W>(s, t, 1, w, m, pos, ipiv + c0, c0);
            if (!ok && t == 0) {
                s_stop = 1;
                atomicExch(&status[kInfo], 1);
            }
            lu_sync<4>(1);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int rl = t + r * 128;
                if (!ok || rl >= m) continue;
                s.perm[c0 + (pos[r] < 0 ? -1 - pos[r] : pos[r])] = (uint16_t)row[r];
                if (pos[r] >= 0) s.lrow[pos[r]] = (uint16_t)rl;
                s_pos[rl] = (int16_t)pos[r];
                s_row[rl] = (uint16_t)row[r];
            }
        }
        __syncthreads();
        if (s_stop) return;
        for (int e = t; e < m * (W / 2); e += kSmThreads) {  // the leaf's columns
            const int rl = e / (W / 2), c = 2 * (e % (W / 2)), j = -1 - s_pos[rl];
            double2 x = *reinterpret_cast<const double2*>(s.S + sx(rl, c));
            if (j >= 0) {
                const double2 u = *reinterpret_cast<const double2*>(s.u + j * W + c);
                x = make_double2(c >= j ? u.x : x.x, c + 1 >= j ? u.y : x.y);
            }
            if (c < w) *reinterpret_cast<double2*>(V + s_row[rl] * ldv + c0 + c) = x;
        }
        auto strips = [&](auto first) {
            for (int q0 = cb + 16 * warp; q0 < n; q0 += 16 * (kSmThreads / 32))
                lu_strip<4, W, decltype(first)::value, true>(s, lane, A, ld, nullptr, n, 0, ldv, V, c0, w, q0);
        };
        if (first) strips(std::true_type{});
        else strips(std::false_type{});
        __syncthreads();
    }
    if (perm)
        for (int i = t; i < n; i += kSmThreads) perm[i] = s.perm[i];
    constexpr int B = 4;
    for (int i0 = warp; i0 < n; i0 += B * (kSmThreads / 32))
        for (int c = lane; c < n; c += 32) {
            double v[B];
#pragma unroll
            for (int q = 0; q < B; ++q) v[q] = V[s.perm[min(i0 + q * (kSmThreads / 32), n - 1)] * ldv + c];
#pragma unroll
            for (int q = 0; q < B; ++q)
                if (i0 + q * (kSmThreads / 32) < n) A[(i0 + q * (kSmThreads / 32)) * ld + c] = v[q];
        }
}

// B <- U^-1 L^-1 P B, eight right-hand sides a CTA: in shared memory, blocks of 32 rows substituted by one
// warp (lane = right-hand side + 8 * (row & 3)) and folded into the others on the FP64 tensor cores.
__global__ void __launch_bounds__(128) small_solve_kernel(const double* LU, int64_t ld, int n, const int32_t* perm,
                                                          double* B, int64_t ldb, int nrhs, const int32_t* status) {
    constexpr int NW = 4, W = 32, NT = 128;
    extern __shared__ __align__(16) unsigned char lu_dyn[];
    LuSlice<NW, W>& s = *reinterpret_cast<LuSlice<NW, W>*>(lu_dyn);
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int q0 = blockIdx.x * kBMaxK, kk = min(kBMaxK, nrhs - q0);
    double* y = s.S;
    for (int i = t; i < n; i += NT) s.perm[i] = (uint16_t)i;
    for (int e = t; e < n * kBMaxK; e += NT) {
        const int j = e / kBMaxK, q = e % kBMaxK;
        y[e] = q < kk ? B[perm[j] * ldb + q0 + q] : 0.0;
    }
    for (int b0 = 0; b0 < n; b0 += W) {
        const int bs = min(W, n - b0);
        __syncthreads();
        batched_copy<NT, 8, double>(t, W * W,  // the block's columns: u[c][r] = L(b0 + r, b0 + c), r > c
            [&](int e) {
                const int r = e / W, c = e % W;
                return (r > c && r < bs) ? LU[(b0 + r) * ld + b0 + c] : 0.0;
            },
            [&](int e, double v) { s.u[e % W * W + e / W] = v; });
        __syncthreads();
        if (warp == 0) {
            const int q = lane & 7, rg = lane >> 3;
            double x[W / 4];
#pragma unroll
            for (int i = 0; i < W / 4; ++i) x[i] = 4 * i + rg < bs ? y[(b0 + 4 * i + rg) * kBMaxK + q] : 0.0;
#pragma unroll 1
            for (int i4 = 0; i4 < W / 4; ++i4) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const double xj = __shfl_sync(0xffffffffu, x[0], q + 8 * v);
                    const double* uc = &s.u[(4 * i4 + v) * W + 4 * i4 + rg];
                    if (rg > v) x[0] = fma(-uc[0], xj, x[0]);
#pragma unroll
                    for (int i = 1; i < W / 4; ++i)
                        if (i4 + i < W / 4) x[i] = fma(-uc[4 * i], xj, x[i]);
                }
                if (4 * i4 + rg < bs) y[(b0 + 4 * i4 + rg) * kBMaxK + q] = x[0];
#pragma unroll
                for (int i = 1; i < W / 4; ++i) x[i - 1] = x[i];
            }
        }
        __syncthreads();
        // the rows below (there are some only below a full block)
        const int g = lane >> 2, tq = lane & 3;
        for (int r0 = b0 + W + 16 * warp; r0 < n; r0 += 16 * NW) {
            const int ra = min(r0 + g, n - 1), rb = min(r0 + g + 8, n - 1);
            double a0[W / 4], a1[W / 4], acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < W / 4; ++k) {
                a0[k] = LU[ra * ld + b0 + 4 * k + tq];
                a1[k] = LU[rb * ld + b0 + 4 * k + tq];
            }
#pragma unroll
            for (int k = 0; k < W / 4; ++k) dmma(acc, a0[k], a1[k], y[(b0 + 4 * k + tq) * kBMaxK + g]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (r0 + g + 8 * e >= n) continue;
                double2* yp = reinterpret_cast<double2*>(y + (r0 + g + 8 * e) * kBMaxK + 2 * tq);
                *yp = make_double2(yp->x - acc[2 * e], yp->y - acc[2 * e + 1]);
            }
        }
    }
    lu_upper<NW, W>(s, t, 1, LU, ld, n);
    __syncthreads();
    for (int e = t; e < n * kBMaxK; e += NT) {
        const int j = e / kBMaxK, q = e % kBMaxK;
        if (q < kk) B[j * ldb + q0 + q] = y[e];
    }
}

template <typename Kern> int32_t small_attr(Ctx* ctx, Kern kern) {
    std::atomic<int>& attr = device_flag((const void*)kern, 0, ctx->device);
    if (!attr.load()) {
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LuSlice<4, 32>)));
        attr.store(1);
    }
    return B2M_OK;
}

size_t batch_smem_bytes(int small_n, int G, int pw_large, int pw_small, int GB) {
    const size_t big = slice_doubles(kBMaxN, pw_large) * ((kBThreads / 32) / GB);
    const size_t small = slice_doubles(small_n, pw_small) * ((kBThreads / 32) / G);
    return std::max(big, small) * sizeof(double);
}

}  // namespace

size_t small_lu_scratch(int64_t n) { return (size_t)(n * ((n + 1) & ~(int64_t)1)) * sizeof(double); }

int32_t small_lu_f64(Ctx* ctx, cudaStream_t st, double* A, int64_t ld, int64_t n, double* V, int32_t* ipiv,
                     int32_t* perm) {
    B2M_TRY(small_attr(ctx, small_lu_kernel));
    prof_begin(ctx, st, kClsPanel);
    small_lu_kernel<<<1, kSmThreads, sizeof(LuSlice<4, 32>), st>>>(A, ld, (int)n, V, ipiv, perm, ctx->d_status);
    prof_end(ctx, st, kClsPanel, 16.0 * n * n);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t small_solve_f64(Ctx* ctx, cudaStream_t st, const double* LU, int64_t ld, int64_t n, const int32_t* perm,
                        double* B, int64_t ldb, int64_t nrhs) {
    B2M_TRY(small_attr(ctx, small_solve_kernel));
    prof_begin(ctx, st, kClsSolve);
    small_solve_kernel<<<(unsigned)ceil_div(nrhs, kBMaxK), 128, sizeof(LuSlice<4, 32>), st>>>(
        LU, ld, (int)n, perm, B, ldb, (int)nrhs, ctx->d_status);
    prof_end(ctx, st, kClsSolve, 0.0);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

// ------------------------------------------------------------------ host side
// A plan's key in the autotuner's table, which saved tables hold.  Different plans may share one (offsets fold into
// each other): it chooses a tile shape, never the data of a call.
static uint64_t plan_signature(int mode, int64_t count, const int32_t* n, const int32_t* k, const int64_t* a_off,
                               const int64_t* b_off) {
    uint64_t sig = 1469598103934665603ull ^ (uint64_t)mode;
    for (int64_t i = 0; i < count; ++i)
        sig = (sig ^ (uint64_t)(n[i] * 16 + k[i]) ^ ((uint64_t)a_off[i] << 20) ^ ((uint64_t)b_off[i] << 40)) *
              1099511628211ull;
    return sig;
}

int32_t batch_solve(Ctx* ctx, cudaStream_t st, int64_t count, const int32_t* hn, const int32_t* hk,
                    const int64_t* ha_off, const int64_t* hb_off, const double* A, const double* B, double* X,
                    int mode, int32_t* info, int32_t* iters, BatchTune* tune_out) {
    if (count <= 0) return B2M_OK;
    if (mode != 0 && mode != 1) return fail(ctx, B2M_ERR_ARG, "batch: mode must be 0 (FP64) or 1 (FP32 + FP64 IR)");
    for (int64_t i = 0; i < count; ++i) {
        if (hn[i] < 1 || hn[i] > kBMaxN) return fail(ctx, B2M_ERR_UNSUPPORTED, "batch: system %lld order %d not in [1, 256]", (long long)i, hn[i]);
        if (hk[i] < 1 || hk[i] > kBMaxK) return fail(ctx, B2M_ERR_UNSUPPORTED, "batch: system %lld has %d right-hand sides (1..8)", (long long)i, hk[i]);
    }
    // device copies of the plan: n, k, offsets, order (largest first), queue head
    const size_t bytes_i = (size_t)count * 4, bytes_l = (size_t)count * 8;
    const size_t plan_bytes = 3 * bytes_i + 2 * bytes_l + 256;
    void* pplan;
    B2M_TRY(ws_get(ctx, kWsPlan, plan_bytes + 256, &pplan));
    char* pp = static_cast<char*>(pplan);
    int32_t* dn = reinterpret_cast<int32_t*>(pp);
    int32_t* dk = dn + count;
    int32_t* dord = dk + count;
    int64_t* dao = reinterpret_cast<int64_t*>(pp + round_up((int64_t)(3 * bytes_i), 256));
    int64_t* dbo = dao + count;
    int32_t* dctr = reinterpret_cast<int32_t*>(dbo + count);
    BatchPlan& plan = ctx->batch_plan;
    if (plan.dev != pplan || plan.n.size() != (size_t)count || std::memcmp(plan.n.data(), hn, bytes_i) != 0 ||
        std::memcmp(plan.k.data(), hk, bytes_i) != 0 || std::memcmp(plan.a_off.data(), ha_off, bytes_l) != 0 ||
        std::memcmp(plan.b_off.data(), hb_off, bytes_l) != 0) {
        std::vector<int32_t> order((size_t)count);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return hn[x] > hn[y]; });
        // the pinned staging buffer may still feed an earlier asynchronous copy
        B2M_CU(ctx, cudaStreamSynchronize(st));
        void* ph = nullptr;
        B2M_TRY(pinned_get(ctx, plan_bytes + 256, &ph));
        char* hp = static_cast<char*>(ph);
        std::memcpy(hp, hn, bytes_i);
        std::memcpy(hp + bytes_i, hk, bytes_i);
        std::memcpy(hp + 2 * bytes_i, order.data(), bytes_i);
        std::memcpy(hp + round_up((int64_t)(3 * bytes_i), 256), ha_off, bytes_l);
        std::memcpy(hp + round_up((int64_t)(3 * bytes_i), 256) + bytes_l, hb_off, bytes_l);
        plan.dev = nullptr;  // (until the copy is enqueued)
        B2M_CU(ctx, cudaMemcpyAsync(pp, hp, round_up((int64_t)(3 * bytes_i), 256) + 2 * bytes_l,
                                    cudaMemcpyHostToDevice, st));
        plan.n.assign(hn, hn + count);
        plan.k.assign(hk, hk + count);
        plan.a_off.assign(ha_off, ha_off + count);
        plan.b_off.assign(hb_off, hb_off + count);
        plan.max_n = hn[order[0]];
        for (int m = 0; m < 2; ++m) plan.sig[m] = plan_signature(m, count, hn, hk, ha_off, hb_off);
        plan.dev = pplan;
    }
    const uint64_t sig = ctx->batch_plan_sig = plan.sig[mode];

    int occ_sms = ctx->num_sms;
    BatchArgs a{};
    a.count = (int)count;
    a.n = dn; a.k = dk; a.a_off = dao; a.b_off = dbo;
    a.A = A; a.B = B; a.X = X;
    a.order = dord; a.counter = dctr; a.info = info; a.iters = iters;
    a.mode = mode;
    a.max_iter = 10;

    auto launch = [&](const BatchTune& tc, cudaStream_t q) -> int32_t {
        const size_t smem = batch_smem_bytes(tc.small_n, tc.group_warps, tc.pw_large, tc.pw_small, tc.big_warps);
        void (*kern)(BatchArgs) = batch_solve_kernel;
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0;
        B2M_CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBThreads, smem));
        if (per_sm < 1) return fail(ctx, B2M_ERR_UNSUPPORTED, "batch: tile shape does not fit one SM");
        const int grid = occ_sms * per_sm;
        void* pscr;
        B2M_TRY(ws_get(ctx, kWsMatD,
                       (size_t)grid * batch_scratch_doubles(tc.small_n, tc.group_warps, tc.big_warps) * sizeof(double),
                       &pscr));
        BatchArgs b = a;
        b.scratch = static_cast<double*>(pscr);
        b.small_n = tc.small_n;
        b.group_warps = tc.group_warps;
        b.big_warps = tc.big_warps;
        b.pw_large = tc.pw_large;
        b.pw_small = tc.pw_small;
        B2M_CU(ctx, cudaMemsetAsync(dctr, 0, sizeof(int32_t), q));
        prof_begin(ctx, q, kClsSolve);
        kern<<<grid, kBThreads, smem, q>>>(b);
        prof_end(ctx, q, kClsSolve, 0.0);
        B2M_LAUNCHED(ctx);
        return B2M_OK;
    };

    // mode 0 has one shape: nothing to tune (the table lists the plan, marked by a negative time)
    auto launch_lu = [&](cudaStream_t q) -> int32_t {
        std::atomic<int>& attr = device_flag((const void*)batch_lu_kernel, 0, ctx->device);
        if (!attr.load()) {
            B2M_CU(ctx, cudaFuncSetAttribute(batch_lu_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(LuShared)));
            attr.store(1);
        }
        const int64_t grid = std::min<int64_t>(count, (int64_t)ctx->num_sms * kLuCtas);
        void* pscr;
        const int64_t per = lu_scratch(plan.max_n);
        B2M_TRY(ws_get(ctx, kWsMatD, (size_t)(grid * per) * sizeof(double), &pscr));
        BatchArgs b = a;
        b.scratch = static_cast<double*>(pscr);
        b.scratch_cta = per;
        B2M_CU(ctx, cudaMemsetAsync(dctr, 0, sizeof(int32_t), q));
        prof_begin(ctx, q, kClsSolve);
        batch_lu_kernel<<<(unsigned)grid, kLuThreads, sizeof(LuShared), q>>>(b, lu_wide(count, ctx->num_sms) ? 1 : 0);
        prof_end(ctx, q, kClsSolve, 0.0);
        B2M_LAUNCHED(ctx);
        return B2M_OK;
    };

    // autotune once per plan (mode, sizes, layout): time each candidate shape on this batch
    BatchTune best;
    auto it = ctx->batch_tunes.find(sig);
    if (it != ctx->batch_tunes.end()) {
        best = it->second;
    } else if (mode == 0) {
        best = ctx->batch_tunes[sig] = BatchTune{64, 1, 32, 16, 8, -1.0f};
    } else {
        std::vector<BatchTune> cands;
        for (int GB : {8, 4})
            for (int pwl : {8, 16, 32})
                for (int G : {1, 2, 4})
                    for (int pws : {8, 16}) cands.push_back(BatchTune{64, G, pwl, pws, GB, 0.0f});
        cudaEvent_t e0, e1;
        B2M_CU(ctx, cudaEventCreate(&e0));
        B2M_CU(ctx, cudaEventCreate(&e1));
        float best_ms = 1e30f;
        for (auto& c : cands) {
            const size_t smem = batch_smem_bytes(c.small_n, c.group_warps, c.pw_large, c.pw_small, c.big_warps);
            if (smem > ctx->smem_optin) continue;
            B2M_TRY(launch(c, st));  // warm
            B2M_CU(ctx, cudaEventRecord(e0, st));
            B2M_TRY(launch(c, st));
            B2M_CU(ctx, cudaEventRecord(e1, st));
            B2M_CU(ctx, cudaEventSynchronize(e1));
            float ms = 0.f;
            B2M_CU(ctx, cudaEventElapsedTime(&ms, e0, e1));
            c.ms = ms;
            if (ms < best_ms) { best_ms = ms; best = c; }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (best_ms >= 1e30f) return fail(ctx, B2M_ERR_UNSUPPORTED, "batch: no tile shape fits");
        ctx->batch_tunes[sig] = best;
    }
    if (tune_out) *tune_out = best;
    // (the launches depend on the plan through its count, its largest order and its tile shape only)
    const GraphKey key{7 + mode * 10, A, B, X, info, count, (int64_t)plan.max_n,
                       best.big_warps * 1000000 + best.pw_large * 10000 + best.pw_small * 100 + best.group_warps,
                       (int64_t)reinterpret_cast<intptr_t>(iters)};
    return run_graph(ctx, st, key, [&](cudaStream_t q) { return mode == 0 ? launch_lu(q) : launch(best, q); });
}

}  // namespace b2m

// ------------------------------------------------------------------ persisted autotuner table
// One text line per batch plan: "<plan signature, hex> <small_n> <group_warps> <pw_large> <pw_small>
// <big_warps> <ms>", after the header line "b2m-batch-tune 2" (a version-1 table, without the
// big_warps column, is read as big_warps = 8).  A later process that loads the table skips the
// timing of the candidate shapes for every plan it lists (the signature covers the mode, every
// system's order, right-hand sides and offsets).  A negative time marks a plan that was not tuned (mode 0): its
// shape is a placeholder that no kernel uses.
extern "C" int32_t b2m_batch_tune_save(b2m_ctx* h, const char* path) {
    b2m::Ctx* ctx = reinterpret_cast<b2m::Ctx*>(h);
    if (!ctx || !path) return B2M_ERR_ARG;
    b2m::CallLock lk(ctx);
    FILE* f = std::fopen(path, "w");
    if (!f) return b2m::fail(ctx, B2M_ERR_ARG, "cannot write %s", path);
    std::fprintf(f, "b2m-batch-tune 2\n");
    for (const auto& e : ctx->batch_tunes)
        std::fprintf(f, "%016llx %d %d %d %d %d %.6f\n", (unsigned long long)e.first, e.second.small_n,
                     e.second.group_warps, e.second.pw_large, e.second.pw_small, e.second.big_warps,
                     (double)e.second.ms);
    return std::fclose(f) == 0 ? B2M_OK : b2m::fail(ctx, B2M_ERR_ARG, "cannot write %s", path);
}

extern "C" int32_t b2m_batch_tune_load(b2m_ctx* h, const char* path, int32_t* loaded) {
    b2m::Ctx* ctx = reinterpret_cast<b2m::Ctx*>(h);
    if (!ctx || !path) return B2M_ERR_ARG;
    b2m::CallLock lk(ctx);
    if (loaded) *loaded = 0;
    FILE* f = std::fopen(path, "r");
    if (!f) return b2m::fail(ctx, B2M_ERR_ARG, "cannot read %s", path);
    char head[32] = {0};
    int version = 0;
    if (std::fscanf(f, "%31s %d", head, &version) != 2 || std::strcmp(head, "b2m-batch-tune") != 0 ||
        (version != 1 && version != 2)) {
        std::fclose(f);
        return b2m::fail(ctx, B2M_ERR_FORMAT, "%s is not a batch tuning table", path);
    }
    unsigned long long sig;
    int sn, g, pwl, pws, gb = 8;
    double ms;
    int n = 0;
    auto next = [&]() -> bool {
        if (version == 1) return std::fscanf(f, "%llx %d %d %d %d %lf", &sig, &sn, &g, &pwl, &pws, &ms) == 6;
        return std::fscanf(f, "%llx %d %d %d %d %d %lf", &sig, &sn, &g, &pwl, &pws, &gb, &ms) == 7;
    };
    while (next()) {
        // only shapes the kernel has: a damaged or foreign line is skipped, never launched
        const bool ok = sn == 64 && (g == 1 || g == 2 || g == 4) && (pwl == 8 || pwl == 16 || pwl == 32) &&
                        (pws == 8 || pws == 16) && (gb == 4 || gb == 8) &&
                        b2m::batch_smem_bytes(sn, g, pwl, pws, gb) <= ctx->smem_optin;
        if (!ok) continue;
        ctx->batch_tunes[(uint64_t)sig] = b2m::BatchTune{sn, g, pwl, pws, gb, (float)ms};
        ++n;
    }
    std::fclose(f);
    if (loaded) *loaded = n;
    return B2M_OK;
}
