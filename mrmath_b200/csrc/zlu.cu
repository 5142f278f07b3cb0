// zlu.cu -- complex (TComplex) LU with partial pivoting, back substitution, solve, inverse and
// determinant on the FP64 building blocks of the real LU.
//
// Reference: InternalRecursiveCplxMatrixLUDecompInPlace (LinAlgLU.pas:1202-1306), CplxLUSwap
// (:1183-1200), CplxLUBacksup (:1147-1181), CplxMatrixLUBackSubst (:1322-1391), CplxMatrixLinEQSolve
// (:1393-1508), CplxMatrixInverseInPlace (:1510-1552), CplxMatrixDeterminant (:1554-1603).  The pivot
// rule is the reference leaf's: the largest CAbs1 = |re| + |im| wins, the first (lowest row) among
// equals, the column is singular when that largest CAbs1 is <= 10/MaxDouble; the column is scaled
// by CInv(pivot) (Smith's formula, CplxSimpleMatrixOperations.pas:288-303) and the pivot placed as
// the reference does; the back substitution divides by U's diagonal with CDiv (:266-285).
//
// B200 design: the interleaved matrix is split into a real and an imaginary plane (row-major, rows
// padded to 128 bytes).  The factorisation is right-looking in leaves of 32 columns, two launches a
// leaf: zpanel_kernel factors it, zstrip_kernel does everything else to the columns outside it
// (interchanges, U12, trailing update).  Matrices wider than kZBlock are split recursively above that, the
// products as four real DMMA GEMMs (Cr -= Ar Br - Ai Bi, Ci -= Ar Bi + Ai Br).  The substitutions
// are the same strip kernel's steps of 32 rows.  The result is interleaved back into the caller's layout.
#include <cooperative_groups.h>

#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"
#include "panel.cuh"

namespace cg = cooperative_groups;

namespace b2m {
namespace {

constexpr int kZLeaf = 32;
constexpr int kZPanelThreads = 1024;
// Widest block without GEMMs.  For the factorisation the line hardly matters (order 2048 took 11.9, 11.3 and 11.3
// ms with 256, 1024 and 4096); solves with many right-hand sides want the GEMMs above it (see zlu_solve).
constexpr int64_t kZBlock = 1024;

struct Planes {
    double* re;
    double* im;
    int64_t ld;
};

__device__ __forceinline__ double2 cinv(double2 x) {
    if (fabs(x.x) >= fabs(x.y)) {
        const double r = x.y / x.x, den = x.x + x.y * r;
        return make_double2(1.0 / den, -r / den);
    }
    const double r = x.x / x.y, den = x.y + r * x.x;
    return make_double2(r / den, -1.0 / den);
}
// x1 - x2 x3 (CSubMul order)
__device__ __forceinline__ double2 csub_mul(double2 x1, double2 x2, double2 x3) {
    return make_double2(x1.x - x2.x * x3.x + x2.y * x3.y, x1.y - x2.x * x3.y - x2.y * x3.x);
}

__global__ void deinterleave_kernel(const double* src, int64_t lws, double* re, double* im, int64_t ld, int64_t rows,
                                    int64_t cols) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= rows * cols) return;
    const int64_t r = e / cols, c = e - r * cols;
    const double2 v = *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(src) + r * lws + c * 16);
    re[r * ld + c] = v.x;
    im[r * ld + c] = v.y;
}

__global__ void interleave_kernel(double* dst, int64_t lwd, const double* re, const double* im, int64_t ld,
                                  int64_t rows, int64_t cols, const int32_t* status) {
    if (status && status[kInfo] != 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= rows * cols) return;
    const int64_t r = e / cols, c = e - r * cols;
    *reinterpret_cast<double2*>(reinterpret_cast<char*>(dst) + r * lwd + c * 16) =
        make_double2(re[r * ld + c], im[r * ld + c]);
}

// (value, row) with the reference's rule: larger value wins, the lower row among equals; -1 = none
__device__ __forceinline__ void best_of(double& a, int& i, double a2, int i2) {
    if (i2 >= 0 && (i < 0 || a2 > a || (a2 == a && i2 < i))) {
        a = a2;
        i = i2;
    }
}

// Leaf factorisation: rows [0, m), columns [0, w) of the planes (P.re/P.im at the panel's origin).
__global__ void __launch_bounds__(kZPanelThreads) zpanel_tall_kernel(Planes P, int m, int w, int row_base, int col_base,
                                                                int32_t* ipiv, int32_t* status) {
    __shared__ double s_a[kZPanelThreads / 32];
    __shared__ int s_i[kZPanelThreads / 32];
    __shared__ double2 s_u[kZLeaf];  // the pivot row after the interchange
    __shared__ int s_piv, s_stop;
    if (status[kInfo] != 0) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_stop = 0;
    for (int j = 0; j < w; ++j) {
        // strict > over rows in ascending order per thread, then the lowest row among equal maxima
        double ba = 0.0;
        int bi = -1;
        for (int i = j + t; i < m; i += kZPanelThreads) {
            const double v = fabs(P.re[(int64_t)i * P.ld + j]) + fabs(P.im[(int64_t)i * P.ld + j]);
            if (v > ba) { ba = v; bi = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double a2 = __shfl_xor_sync(0xffffffffu, ba, o);
            const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
            best_of(ba, bi, a2, i2);
        }
        if (lane == 0) { s_a[warp] = ba; s_i[warp] = bi; }
        __syncthreads();
        if (warp == 0) {
            ba = s_a[lane];
            bi = s_i[lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double a2 = __shfl_xor_sync(0xffffffffu, ba, o);
                const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
                best_of(ba, bi, a2, i2);
            }
            if (lane == 0) {
                s_piv = bi;
                if (bi < 0 || !(ba > 10.0 / DBL_MAX)) {
                    s_stop = 1;
                    atomicExch(&status[kInfo], 1);
                } else {
                    ipiv[col_base + j] = row_base + bi;
                }
            }
        }
        __syncthreads();
        if (s_stop) return;
        const int p = s_piv;
        // interchange rows j and p over the panel's columns; keep the pivot row for the update
        if (t < w) {
            const int64_t oj = (int64_t)j * P.ld + t, op = (int64_t)p * P.ld + t;
            const double2 vj = make_double2(P.re[oj], P.im[oj]), vp = make_double2(P.re[op], P.im[op]);
            s_u[t] = vp;
            if (p != j) {
                P.re[oj] = vp.x; P.im[oj] = vp.y;
                P.re[op] = vj.x; P.im[op] = vj.y;
            }
        }
        __syncthreads();
        const double2 s = cinv(s_u[j]);
        for (int i = j + 1 + t; i < m; i += kZPanelThreads) {
            const int64_t o = (int64_t)i * P.ld;
            const double2 x = make_double2(P.re[o + j], P.im[o + j]);
            // CAddMul(0, x, s): 0 + x.re s.re - x.im s.im, 0 + x.re s.im + x.im s.re
            const double2 l = make_double2(0.0 + x.x * s.x - x.y * s.y, 0.0 + x.x * s.y + x.y * s.x);
            P.re[o + j] = l.x;
            P.im[o + j] = l.y;
            for (int k = j + 1; k < w; ++k) {
                const double2 a = make_double2(P.re[o + k], P.im[o + k]);
                const double2 r = csub_mul(a, l, s_u[k]);
                P.re[o + k] = r.x;
                P.im[o + k] = r.y;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// Leaf of up to 32 columns and 4096 rows on a cluster of up to 16 CTAs: the elimination of panel.cu's
// panel_kernel (rows never move; eight columns at a time in registers that shift left by one a column;
// each warp sends its candidate to every CTA; leading words decide, exact comparison on ties) with
// complex elements, without the scribe warp: two candidate slots are enough, since a warp sends
// column j + 2 only after every warp has sent column j + 1 and so has left column j.
// map[i] (absolute rows, of the panel's rows) receives the row whose content ends in row i.
// Chain of a column, 1,850 cycles in a cluster: update, CInv of every lane's best value under the warp
// reduction and the sending, 800; the exchange, 740; selection, 310.  1,350 on a lone CTA, whose candidates stay
// in its own shared memory.  (Choosing a CTA's candidate before the exchange, to send a quarter of the bytes,
// was slower: 45 us a leaf instead of 41.)  Measured on a B200, 32 columns: 600 rows 932 us (one CTA of 1024 threads,
// rows in L2) -> 40 us; 160 rows 36 us, 64 rows 24 us.
// ------------------------------------------------------------------------------------------
constexpr int kZNw = 4;            // warps
constexpr int kZNt = kZNw * 32;
constexpr int kZBk = 8;            // columns per block
constexpr int kZMaxC = 16;         // largest cluster

struct __align__(16) ZCand {
    double2 rinv;      // CInv(row[0])
    double mag;        // CAbs1(row[0]); 0: no candidate
    int pos, lrow;     // position in the panel, local row of its CTA
    double2 row[kZBk];  // the row's block columns, from the current one on
};
static_assert(sizeof(ZCand) == 160, "ten 16-byte pieces");

// 16-byte pieces of a candidate of column `col` that the rest of its block can use
__device__ __forceinline__ int zcand_pieces(int col) { return 2 + kZBk - (col & (kZBk - 1)); }

__device__ __forceinline__ uint4 zbits(double2 v) {
    const unsigned long long x = __double_as_longlong(v.x), y = __double_as_longlong(v.y);
    return make_uint4((uint32_t)x, (uint32_t)(x >> 32), (uint32_t)y, (uint32_t)(y >> 32));
}

// CInv of v without a divergent branch; any: the lane has a value (else 1, by an opaque select, so that
// nothing divides by zero, whose slow path would cost the whole warp)
__device__ __forceinline__ double2 cinv_lane(double2 v, bool any) {
    double x, y;
    asm("{ .reg .pred p; setp.ne.u32 p, %4, 0; selp.f64 %0, %2, 0d3FF0000000000000, p; "
        "selp.f64 %1, %3, 0d3FF0000000000000, p; }"
        : "=d"(x), "=d"(y)
        : "d"(v.x), "d"(v.y), "r"(any ? 1 : 0));
    const bool re = fabs(x) >= fabs(y);
    const double big = re ? x : y, sm = re ? y : x;
    // (quotients as the product with the reciprocal, corrected by the exact residual: 220 cycles instead of 360
    // on the chain; by divisions where an operand is far from 1)
    double r, ri, i;
    const double ib = 1.0 / big;
    r = sm * ib;
    r = fma(fma(-r, big, sm), ib, r);
    double den = big + sm * r;
    i = 1.0 / den;
    ri = r * i;
    ri = fma(fma(-ri, den, r), i, ri);
    if (mag_hi(big) - 0x03700000u >= 0x79000000u) {  // outside 2^-968 .. 2^968 (|r| <= 1, |den| <= 2 |big|)
        r = sm / big;
        den = big + sm * r;
        i = 1.0 / den;
        ri = r / den;
    }
    return re ? make_double2(i, -ri) : make_double2(ri, -i);
}

template <int RPT, bool MULTI>
__global__ void __launch_bounds__(kZNt, 1)
    zpanel_kernel(Planes P, int m, int w, int R, int row_base, int32_t* ipiv, int32_t* map, int32_t* status,
                  uint32_t polls) {
    int C = 1, rank = 0;
    if constexpr (MULTI) {
        C = (int)cg::this_cluster().num_blocks();
        rank = (int)cg::this_cluster().block_rank();
    }
    extern __shared__ __align__(16) double2 Z[];  // this CTA's rows [R][32], elements swizzled by row
    auto sx = [](int row, int c) -> int { return row * kZLeaf + (c ^ (row & 7)); };
    constexpr int kNone = kZNw * kZMaxC;  // (no candidate: mag 0)
    __shared__ ZCand s_loc[2][kZNw], s_rcv[2][kNone + 1];
    __shared__ __align__(16) double2 s_u[kZLeaf][kZLeaf], s_l[kZBk][kZBk];
    __shared__ __align__(16) uint32_t s_key[2][kZNw];  // leading words of a lone CTA's candidates
    __shared__ __align__(8) uint64_t s_bar[2], s_rbar;
    __shared__ int s_pl[kZLeaf], s_ps[kZLeaf];
    __shared__ int s_late;  // a wait of the cluster ran out
    if (status[kInfo] != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lo = rank * R, nr = max(0, min(m, lo + R) - lo);
    if (MULTI && tid == 0) {
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        mbar_init(&s_rbar, 1);
        s_late = 0;
        s_rcv[0][kNone].mag = s_rcv[1][kNone].mag = 0.0;
        fence_barrier_init();
        for (int j = 0; j < min(2, w); ++j)
            mbar_arrive_expect_tx(&s_bar[j], (uint32_t)(C * kZNw * 16 * zcand_pieces(j)));
        mbar_arrive_expect_tx(&s_rbar, (uint32_t)(kZBk * kZLeaf * 16));
    }
    __syncwarp();
    if constexpr (MULTI) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
#pragma unroll 4
    for (int e = tid; e < nr * kZLeaf; e += kZNt) {
        const int rl = e / kZLeaf, c = e % kZLeaf;
        const int64_t o = (int64_t)(lo + rl) * P.ld + (c < w ? c : 0);
        cp_async8(&Z[sx(rl, c)].x, P.re + o, c < w ? 8 : 0);
        cp_async8(&Z[sx(rl, c)].y, P.im + o, c < w ? 8 : 0);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if constexpr (MULTI) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    bool late = false;  // this thread, after select() some thread of its warp, gave up a wait (see panel.cuh)
    // the pivot of a column among the cluster's candidates, the same in every warp (kNone for a warp that is late)
    auto select = [&](const ZCand* cands) -> int {
        if constexpr (!MULTI) {
            const uint4 kv = *reinterpret_cast<const uint4*>(&s_key[cands == s_rcv[1] ? 1 : 0][0]);
            const uint32_t k[kZNw] = {kv.x, kv.y, kv.z, kv.w};
            const uint32_t M = max(max(k[0], k[1]), max(k[2], k[3]));
            int n = 0, win = 0;
#pragma unroll
            for (int q = kZNw - 1; q >= 0; --q) {
                win = k[q] == M ? q : win;
                n += k[q] == M ? 1 : 0;
            }
            if (n > 1) {
                win = warp_winner(lane < kZNw ? cands[lane].mag : 0.0, lane < kZNw ? cands[lane].pos : 0x7fffffff);
                if (win >= kZNw) win = 0;
            }
            return win;
        }
        const int cnt = C * kZNw;
        uint32_t k[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) k[e] = lane + 32 * e < cnt ? mag_hi(cands[lane + 32 * e].mag) : 0u;
        const uint32_t mk = max(k[0], k[1]);
        int q = k[0] == mk ? lane : lane + 32;
        const uint32_t M = __reduce_max_sync(0xffffffffu, mk);
        const uint32_t bal = __ballot_sync(0xffffffffu, mk == M);
        const uint32_t bal2 = __ballot_sync(0xffffffffu, late || (mk == M && k[0] == k[1]));
        int wl = __ffs(bal) - 1;
        if ((bal & (bal - 1)) || bal2) {
            late = __any_sync(0xffffffffu, late);
            if (late) return kNone;
            double ba = 0.0;
            int bp = 0x7fffffff;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (lane + 32 * e >= cnt) continue;
                const double a = cands[lane + 32 * e].mag;
                const int p = cands[lane + 32 * e].pos;
                if (a > ba || (a == ba && p < bp)) { ba = a; bp = p; q = lane + 32 * e; }
            }
            wl = warp_winner(ba, bp);
        }
        const uint32_t odd = __ballot_sync(0xffffffffu, q >= 32);
        const int win = wl + (((odd >> wl) & 1u) ? 32 : 0);
        return win < cnt ? win : 0;
    };
    auto wait_bar = [&](uint64_t* bar, const uint32_t phase, const int site) {
        late = !cluster_wait(bar, phase, polls, &s_late, C, status, site);
    };
    int pos[RPT];
    double2 act[RPT][kZBk];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int rl = tid + r * kZNt;
        pos[r] = rl < nr ? lo + rl : -1 - kZLeaf;
#pragma unroll
        for (int i = 0; i < kZBk; ++i) act[r][i] = rl < nr ? Z[sx(rl, i)] : make_double2(0.0, 0.0);
    }
    // lane l sends to CTA l % C of the cluster, pieces l / C, l / C + 32 / C, ...
    const int push_q = lane / C, push_step = 32 / C;
    uint32_t push_dst = 0, push_bar = 0;
    if constexpr (MULTI) {
        push_dst = map_rank(&s_rcv[0][rank * kZNw + warp], lane % C);
        push_bar = map_rank(&s_bar[0], lane % C);
    }
    auto publish = [&](const int col) {
        const int slot = col & 1;
        double mg[RPT];
        uint32_t h[RPT], mh = 0;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            mg[r] = pos[r] >= 0 ? fabs(act[r][0].x) + fabs(act[r][0].y) : 0.0;
            h[r] = mag_hi(mg[r]);
            mh = max(mh, h[r]);
        }
        double2 cr[kZBk];
        double ba = mg[0];
        int cp = pos[0], cl = tid, cnt = h[0] == mh ? 1 : 0;
#pragma unroll
        for (int i = 0; i < kZBk; ++i) cr[i] = act[0][i];
#pragma unroll
        for (int r = 1; r < RPT; ++r) {
            const bool is = h[r] == mh;
            cnt += is ? 1 : 0;
#pragma unroll
            for (int i = 0; i < kZBk; ++i) {
                cr[i].x = is ? act[r][i].x : cr[i].x;
                cr[i].y = is ? act[r][i].y : cr[i].y;
            }
            ba = is ? mg[r] : ba;
            cp = is ? pos[r] : cp;
            cl = is ? tid + r * kZNt : cl;
        }
        double2 rinv = cinv_lane(cr[0], mh != 0);
        const uint32_t M = __reduce_max_sync(0xffffffffu, mh);
        const uint32_t b1 = __ballot_sync(0xffffffffu, mh == M);
        const uint32_t b2 = __ballot_sync(0xffffffffu, mh == M && cnt > 1);
        int wl = __ffs(b1) - 1;
        if (M != 0 && ((b1 & (b1 - 1)) || b2 || M >= kInfHi)) {  // ties and values that are not finite: exactly
            ba = 0.0;
            cp = 0x7fffffff;
#pragma unroll
            for (int r = 0; r < RPT; ++r)
                if (pos[r] >= 0 && mg[r] > 0.0 && (mg[r] > ba || (mg[r] == ba && pos[r] < cp))) {
                    ba = mg[r];
                    cp = pos[r];
                    cl = tid + r * kZNt;
#pragma unroll
                    for (int i = 0; i < kZBk; ++i) cr[i] = act[r][i];
                }
            rinv = cinv_lane(cr[0], ba > 0.0);
            wl = warp_winner(ba, cp);
        }
        if (lane == wl) {
            ZCand& c = MULTI ? s_loc[slot][warp] : s_rcv[slot][warp];
#pragma unroll
            for (int i = 0; i < kZBk; ++i) c.row[i] = cr[i];
            c.rinv = rinv;
            c.mag = M != 0 ? ba : 0.0;
            if (!MULTI) s_key[slot][warp] = mag_hi(c.mag);
            *reinterpret_cast<int2*>(&c.pos) = make_int2(M != 0 ? cp : 0x7fffffff, cl);
        }
        if constexpr (MULTI) {
            __syncwarp();
            const uint4* src = reinterpret_cast<const uint4*>(&s_loc[slot][warp]);
            const int np = zcand_pieces(col);
            if (push_q < push_step)
                for (int q = push_q; q < np; q += push_step)
                    st_async16(push_dst + slot * (uint32_t)sizeof(s_rcv[0]) + 16 * q, src[q], push_bar + 8 * slot);
        }
    };
    bool dead = false;  // this warp met a singular column or is late; the CTA leaves at its next common barrier
    bool left = false;  // it has left
    publish(0);
    for (int jb = 0; jb < w; jb += kZBk) {
        const int bw = min(kZBk, w - jb);
#pragma unroll 1
        for (int t = 0; t < bw; ++t) {
            const int j = jb + t;
            if constexpr (MULTI) wait_bar(&s_bar[j & 1], (j >> 1) & 1, 204);
            else __syncthreads();
            if (MULTI && tid == 0 && !late && j + 2 < w)
                mbar_arrive_expect_tx(&s_bar[j & 1], (uint32_t)(C * kZNw * 16 * zcand_pieces(j + 2)));
            const int win = select(s_rcv[j & 1]);
            const ZCand& b = s_rcv[j & 1][win];
            double2 u[kZBk];
#pragma unroll
            for (int i = 0; i < kZBk; ++i) u[i] = b.row[i];
            const double2 rinv = b.rinv;
            const int2 pl = *reinterpret_cast<const int2*>(&b.pos);
            if (!(b.mag > 10.0 / DBL_MAX)) {
                if (rank == 0 && tid == 0 && !late) atomicExch(&status[kInfo], 1);
                dead = true;
                break;
            }
            const bool mine = MULTI ? win / kZNw == rank : true;
            if (warp == kZNw - 1) {  // the pivot, and its row's part of U inside its block
                if (lane < kZBk - t && j + lane < kZLeaf) s_u[j][j + lane] = b.row[lane];
                if (lane == 0) {
                    if (rank == 0) ipiv[row_base + j] = row_base + pl.x;
                    s_pl[j] = pl.y;
                    s_ps[j] = MULTI ? win / kZNw : 0;
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int rl = tid + r * kZNt;
                if (mine && rl == pl.y) pos[r] = -1 - j;
                else if (pos[r] == j) pos[r] = pl.x;
                // CAddMul(0, x, s): 0 + x.re s.re - x.im s.im, 0 + x.re s.im + x.im s.re
                const double2 x = act[r][0];
                const double2 l = make_double2(0.0 + x.x * rinv.x - x.y * rinv.y, 0.0 + x.x * rinv.y + x.y * rinv.x);
                if (pos[r] >= 0) Z[sx(rl, j)] = l;
#pragma unroll
                for (int i = 1; i < kZBk; ++i) act[r][i - 1] = csub_mul(act[r][i], l, u[i]);
                act[r][kZBk - 1] = make_double2(0.0, 0.0);
            }
            if (t + 1 < bw) publish(j + 1);
        }
        // ---- block end: the pivot rows as their owners hold them (multipliers, and the columns right
        // of the block without the block's updates) come together in every CTA
        const int c1 = jb + kZBk;
        if (c1 >= w) break;
        left = __syncthreads_or(dead);
        if (left) break;
        for (int e = tid; e < kZBk * kZLeaf; e += kZNt) {
            const int t = e / kZLeaf, c = e % kZLeaf;
            if (s_ps[jb + t] == rank && c >= jb) {
                const double2 v = Z[sx(s_pl[jb + t], c)];
                double2* dst = c >= c1 ? &s_u[jb + t][c] : &s_l[t][c - jb];
                if constexpr (MULTI) {
                    for (int d = 0; d < C; ++d) st_async16(map_rank(dst, d), zbits(v), map_rank(&s_rbar, d));
                } else {
                    *dst = v;
                }
            }
        }
        if constexpr (MULTI) wait_bar(&s_rbar, (jb / kZBk) & 1, 205);
        else __syncthreads();
        if (warp == 0 && c1 + lane < kZLeaf) {
            const int c = c1 + lane;
            double2 x[kZBk];
#pragma unroll
            for (int q = 0; q < kZBk; ++q) x[q] = s_u[jb + q][c];
#pragma unroll
            for (int t0 = 0; t0 < kZBk - 1; ++t0)
#pragma unroll
                for (int t1 = t0 + 1; t1 < kZBk; ++t1) x[t1] = csub_mul(x[t1], s_l[t1][t0], x[t0]);
#pragma unroll
            for (int q = 1; q < kZBk; ++q) s_u[jb + q][c] = x[q];
        }
        if (MULTI && tid == 0 && !late) mbar_arrive_expect_tx(&s_rbar, (uint32_t)(kZBk * (kZLeaf - c1) * 16));
        left = __syncthreads_or(late);
        if (left) break;
#pragma unroll 1
        for (int c = c1; c < kZLeaf; c += 4) {  // four columns a step; the first eight stay in registers
            double2 x[RPT][4];
#pragma unroll
            for (int r = 0; r < RPT; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    x[r][i] = pos[r] >= 0 ? Z[sx(tid + r * kZNt, c + i)] : make_double2(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < kZBk; ++q) {
                double2 l[RPT];
#pragma unroll
                for (int r = 0; r < RPT; ++r)
                    l[r] = pos[r] >= 0 ? Z[sx(tid + r * kZNt, jb + q)] : make_double2(0.0, 0.0);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double2 uu = s_u[jb + q][c + i];
#pragma unroll
                    for (int r = 0; r < RPT; ++r) x[r][i] = csub_mul(x[r][i], l[r], uu);
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (pos[r] >= 0) Z[sx(tid + r * kZNt, c + i)] = x[r][i];
            if (c == c1 + 4) {  // the next block is complete: its first candidates go out under the rest
#pragma unroll
                for (int r = 0; r < RPT; ++r)
#pragma unroll
                    for (int i = 0; i < kZBk; ++i)
                        act[r][i] = pos[r] >= 0 ? Z[sx(tid + r * kZNt, c1 + i)] : make_double2(0.0, 0.0);
                publish(c1);
            }
        }
    }
    if (!left) left = __syncthreads_or(dead);
    if (!left) {
        // every row goes to its position: rows below the pivots as they are (multipliers), the pivot
        // rows held here with U from the diagonal on
        int* s_pos = reinterpret_cast<int*>(&s_loc[0][0]);
        static_assert(sizeof(s_loc) >= (size_t)kZNt * RPT * sizeof(int), "positions fit");
#pragma unroll
        for (int r = 0; r < RPT; ++r) s_pos[tid + r * kZNt] = pos[r];
        __syncthreads();
        constexpr int B = 8;  // rows a step, their loads together
        for (int r0 = warp; r0 < nr; r0 += B * kZNw) {
            int fin[B];
            double2 v[B];
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const int rl = min(r0 + q * kZNw, nr - 1), ps = s_pos[rl];
                fin[q] = ps >= 0 ? ps : -1 - ps;
                v[q] = *(ps < 0 && lane >= fin[q] ? &s_u[fin[q] & (kZLeaf - 1)][lane] : &Z[sx(rl, lane)]);
            }
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const bool ok = fin[q] < m && r0 + q * kZNw < nr;
                double* dr = P.re + (int64_t)fin[q] * P.ld + lane;
                double* di = P.im + (int64_t)fin[q] * P.ld + lane;
                if (ok && lane < w) *dr = v[q].x;
                if (ok && lane < w) *di = v[q].y;
                if (ok && lane == 0) map[row_base + fin[q]] = row_base + lo + r0 + q * kZNw;
            }
        }
    }
    if constexpr (MULTI) cluster_leave(&s_late);
}

// ------------------------------------------------------------------------------------------
// One step of 32 rows [r0, r0 + k) with their triangle T(r0.., r0..): on columns [xlo, xhi) of X the
// rows are solved (unit lower or, kUpper, upper with T's diagonal) and rows [u0, u1) -= T(rows, r0..) times
// them.  With map (a leaf's interchanges, see zpanel_kernel; u0 = r0 + k, u1 = n) every row is first
// replaced by row map[row], also in the columns [0, left) and [right, end), which are not solved, and perm
// likewise.  Solved rows go to Y (Y.re null: in place; not in place when gridDim.y > 1, since every CTA
// of a strip solves the step for itself).
//
// A CTA takes eight columns: one warp a column for the triangle (lane = row, shuffles), then 16 x 8
// tiles of the rows below on the FP64 tensor cores, real and imaginary part as two 16 x 8
// accumulators.  The interchanges need no other CTA's rows: a row outside the step receives only rows
// of the step, which are kept in shared memory before anything is written.  A strip of eight is
// what keeps 148 SMs busy at order 600 (71 strips of the first leaf); with it the interchanges, U12 and the update
// of a leaf take 14 us on average (before: two launches of interchanges, one triangular solve and four
// GEMMs, 88 us).  Order 600 with two right-hand sides from host memory: 19.0 ms before, 1.64 ms now.
// ------------------------------------------------------------------------------------------
constexpr int kZsThreads = 256;
constexpr int kZsCols = 8;
static_assert(kZsCols == kZsThreads / 32, "a warp a column");

struct ZStrip {
    Planes T, X, Y;
    int r0, k, u0, u1;
    int xlo, xhi, left, right, end;
    int nsolve, nleft, nright;  // strips
    const int32_t* map;
    int32_t* perm;
    const int32_t* status;
};

template <bool kUpper> __global__ void __launch_bounds__(kZsThreads, 2) zstrip_kernel(ZStrip a) {
    __shared__ double2 s_t[kZLeaf][kZLeaf + 1], s_x[kZLeaf][kZsCols + 1], s_top[kZLeaf][kZsCols + 1];
    if (a.status[kInfo] != 0 || a.status[kTimeout] != 0) return;  // (map is not complete after a wait that ran out)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.x;
    const int r0 = a.r0, k = a.k;
    if (b >= a.nsolve + a.nleft + a.nright) {  // perm
        int* s_p = reinterpret_cast<int*>(&s_top[0][0]);
        int src = 0;
        if (tid < k) {
            s_p[tid] = a.perm[r0 + tid];
            src = a.perm[a.map[r0 + tid]];
        }
        __syncthreads();
        if (tid < k) a.perm[r0 + tid] = src;
        for (int i = a.u0 + tid; i < a.u1; i += kZsThreads) {
            const int q = a.map[i];
            if (q != i) a.perm[i] = s_p[q - r0];
        }
        return;
    }
    const bool solve = b < a.nsolve;
    const int x0 = solve ? a.xlo + b * kZsCols
                         : (b < a.nsolve + a.nleft ? (b - a.nsolve) * kZsCols
                                                   : a.right + (b - a.nsolve - a.nleft) * kZsCols);
    const int xe = solve ? a.xhi : (b < a.nsolve + a.nleft ? a.left : a.end);
    const int64_t ldx = a.X.ld, ldt = a.T.ld;
    const int col = x0 + warp;
    const bool in = lane < k && col < xe;
    double2 x = make_double2(0.0, 0.0);
    if (in) {
        const int64_t o = (int64_t)(r0 + lane) * ldx + col;
        if (a.map) {
            s_top[lane][warp] = make_double2(a.X.re[o], a.X.im[o]);
            const int64_t q = (int64_t)a.map[r0 + lane] * ldx + col;
            x = make_double2(a.X.re[q], a.X.im[q]);
        } else {
            x = make_double2(a.X.re[o], a.X.im[o]);
        }
    }
    if (!solve) {  // interchanges only
        __syncthreads();
        if (in) {
            a.X.re[(int64_t)(r0 + lane) * ldx + col] = x.x;
            a.X.im[(int64_t)(r0 + lane) * ldx + col] = x.y;
        }
        for (int i = a.u0 + tid; i < a.u1; i += kZsThreads) {
            const int q = a.map[i];
            if (q == i) continue;
            for (int c = 0; c < kZsCols && x0 + c < xe; ++c) {
                a.X.re[(int64_t)i * ldx + x0 + c] = s_top[q - r0][c].x;
                a.X.im[(int64_t)i * ldx + x0 + c] = s_top[q - r0][c].y;
            }
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < kZLeaf * kZLeaf / kZsThreads; ++e) {
        const int row = warp + e * (kZsThreads / 32);
        const int64_t o = (int64_t)(r0 + row) * ldt + r0 + lane;
        s_t[row][lane] = row < k && lane < k ? make_double2(a.T.re[o], a.T.im[o]) : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if constexpr (!kUpper) {
#pragma unroll 8
        for (int j = 0; j < kZLeaf - 1; ++j) {  // (zero multipliers past k)
            const double2 xj = make_double2(__shfl_sync(0xffffffffu, x.x, j), __shfl_sync(0xffffffffu, x.y, j));
            if (lane > j) x = csub_mul(x, s_t[lane][j], xj);
        }
    } else {
        // CDiv by the row's diagonal: its ratio and denominator once a lane, then the product with the
        // reciprocal corrected by the exact residual; with divisions where the denominator is far from 1
        // or a result is not finite
        const double2 d = lane < k ? s_t[lane][lane] : make_double2(1.0, 0.0);
        const bool re = fabs(d.x) >= fabs(d.y);
        const double big = re ? d.x : d.y, r = (re ? d.y : d.x) / big, den = big + (re ? d.y : d.x) * r;
        const double inv = 1.0 / den;
        const double2 xs = x;
        auto sweep = [&](auto divide) {
            x = xs;
#pragma unroll 4
            for (int j = kZLeaf - 1; j >= 0; --j) {
                if (j >= k) continue;
                double nx = re ? x.x + r * x.y : x.x * r + x.y, ny = re ? x.y - r * x.x : x.y * r - x.x;
                if constexpr (decltype(divide)::value) {
                    nx /= den;
                    ny /= den;
                } else {
                    const double qx = nx * inv, qy = ny * inv;
                    nx = fma(fma(-qx, den, nx), inv, qx);
                    ny = fma(fma(-qy, den, ny), inv, qy);
                }
                const double2 xj = make_double2(__shfl_sync(0xffffffffu, nx, j), __shfl_sync(0xffffffffu, ny, j));
                if (lane == j) x = xj;
                else if (lane < j) x = csub_mul(x, s_t[lane][j], xj);
            }
        };
        const uint32_t dh = mag_hi(den);
        bool again = __any_sync(0xffffffffu, dh - 0x01700000u >= 0x7d000000u);  // outside 2^-1000 .. 2^1000
        if (!again) {
            sweep(std::false_type{});
            again = __any_sync(0xffffffffu, mag_hi(x.x) >= kInfHi || mag_hi(x.y) >= kInfHi);
        }
        if (again) sweep(std::true_type{});
    }
    s_x[lane][warp] = x;
    if (in && (a.Y.re == nullptr || blockIdx.y == 0)) {
        const Planes& Y = a.Y.re ? a.Y : a.X;
        Y.re[(int64_t)(r0 + lane) * Y.ld + col] = x.x;
        Y.im[(int64_t)(r0 + lane) * Y.ld + col] = x.y;
    }
    __syncthreads();
    // m16n8k4 fragments: a = T[g][k], T[g + 8][k], b = x[k][g], c = rows g, g + 8, columns 2t, 2t + 1;
    // step (q, s) takes the k's 8 q + 2 t + s, so that T's are read as pairs
    const int g = lane >> 2, t = lane & 3;
    double nre[kZLeaf / 4], pim[kZLeaf / 4], nim[kZLeaf / 4];
#pragma unroll
    for (int q = 0; q < kZLeaf / 8; ++q)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double2 v = s_x[8 * q + 2 * t + s][g];
            nre[2 * q + s] = -v.x;
            pim[2 * q + s] = v.y;
            nim[2 * q + s] = -v.y;
        }
    auto mma = [](double (&d)[4], double a0, double a1, double bb) {
        asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                     : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                     : "d"(a0), "d"(a1), "d"(bb));
    };
    const int c = x0 + 2 * t;
#pragma unroll 1
    for (int t0 = a.u0 + 16 * (warp + (kZsThreads / 32) * blockIdx.y); t0 < a.u1;
         t0 += 16 * (kZsThreads / 32) * gridDim.y) {
        const int row[2] = {min(t0 + g, a.u1 - 1), min(t0 + g + 8, a.u1 - 1)};
        double ar[4] = {}, ai[4] = {};
        double2 lr[2][kZLeaf / 8], li[2][kZLeaf / 8];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int q = 0; q < kZLeaf / 8; ++q) {
                const int64_t o = (int64_t)row[e] * ldt + r0 + 8 * q + 2 * t;
                double2 vr = make_double2(0.0, 0.0), vi = vr;
                if (8 * q + 2 * t < k) {
                    vr = *reinterpret_cast<const double2*>(a.T.re + o);
                    vi = *reinterpret_cast<const double2*>(a.T.im + o);
                    if (8 * q + 2 * t + 1 >= k) vr.y = vi.y = 0.0;
                }
                lr[e][q] = vr;
                li[e][q] = vi;
            }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int q = a.map ? a.map[row[e]] : row[e];
            if (c >= xe) continue;
            if (q != row[e]) {
                const double2 v0 = s_top[q - r0][2 * t], v1 = c + 1 < xe ? s_top[q - r0][2 * t + 1] : v0;
                ar[2 * e] = v0.x; ar[2 * e + 1] = v1.x;
                ai[2 * e] = v0.y; ai[2 * e + 1] = v1.y;
            } else {
                const double2 vr = *reinterpret_cast<const double2*>(a.X.re + (int64_t)q * ldx + c);
                const double2 vi = *reinterpret_cast<const double2*>(a.X.im + (int64_t)q * ldx + c);
                ar[2 * e] = vr.x; ar[2 * e + 1] = vr.y;
                ai[2 * e] = vi.x; ai[2 * e + 1] = vi.y;
            }
        }
#pragma unroll
        for (int q = 0; q < kZLeaf / 8; ++q) {
            mma(ar, lr[0][q].x, lr[1][q].x, nre[2 * q]);
            mma(ai, lr[0][q].x, lr[1][q].x, nim[2 * q]);
            mma(ar, li[0][q].x, li[1][q].x, pim[2 * q]);
            mma(ai, li[0][q].x, li[1][q].x, nre[2 * q]);
            mma(ar, lr[0][q].y, lr[1][q].y, nre[2 * q + 1]);
            mma(ai, lr[0][q].y, lr[1][q].y, nim[2 * q + 1]);
            mma(ar, li[0][q].y, li[1][q].y, pim[2 * q + 1]);
            mma(ai, li[0][q].y, li[1][q].y, nre[2 * q + 1]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (t0 + g + 8 * e >= a.u1 || c >= xe) continue;
            double* dr = a.X.re + (int64_t)row[e] * ldx + c;
            double* di = a.X.im + (int64_t)row[e] * ldx + c;
            if (c + 1 < xe) {
                *reinterpret_cast<double2*>(dr) = make_double2(ar[2 * e], ar[2 * e + 1]);
                *reinterpret_cast<double2*>(di) = make_double2(ai[2 * e], ai[2 * e + 1]);
            } else {
                *dr = ar[2 * e];
                *di = ai[2 * e];
            }
        }
    }
}

// X[i][:] = B[perm[i]][:] on both planes
__global__ void zgather_rows_kernel(double* xre, double* xim, int64_t ldx, const double* bre, const double* bim,
                                    int64_t ldb, const int32_t* perm, int64_t n, int64_t nrhs) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * nrhs) return;
    const int64_t i = e / nrhs, c = e - i * nrhs;
    xre[i * ldx + c] = bre[(int64_t)perm[i] * ldb + c];
    xim[i * ldx + c] = bim[(int64_t)perm[i] * ldb + c];
}

// det = (+-1, 0) * U[0][0] * U[1][1] * ... in order (CMul), 1024 threads
__global__ void __launch_bounds__(1024) zdeterminant_kernel(Planes P, int n, const int32_t* ipiv,
                                                            const int32_t* status, double* det) {
    __shared__ double2 dg[1024];
    __shared__ int flips;
    if (threadIdx.x == 0) flips = 0;
    __syncthreads();
    int local = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (ipiv[i] != i) local++;
    atomicAdd(&flips, local);
    __syncthreads();
    double2 r = make_double2((flips & 1) ? -1.0 : 1.0, 0.0);
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int i = c0 + (int)threadIdx.x;
        if (i < n) dg[threadIdx.x] = make_double2(P.re[(int64_t)i * P.ld + i], P.im[(int64_t)i * P.ld + i]);
        __syncthreads();
        if (threadIdx.x == 0) {
            const int cnt = min(1024, n - c0);
            for (int k = 0; k < cnt; ++k) {
                const double2 b = dg[k];
                r = make_double2(r.x * b.x - r.y * b.y, r.x * b.y + r.y * b.x);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const bool sing = status[kInfo] != 0;
        det[0] = sing ? 0.0 : r.x;
        det[1] = sing ? 0.0 : r.y;
    }
}

unsigned zblocks(int64_t e) { return (unsigned)ceil_div(std::max<int64_t>(e, 1), 256); }

__global__ void ziota_kernel(int32_t* v, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (int32_t)i;
}

// C (M x N at c0 of both planes) -= A (M x K) B (K x N) as four real DMMA GEMMs
int32_t zgemm_sub(Ctx* ctx, cudaStream_t st, const Planes& Ap, int64_t an, int64_t ar0, int64_t ac0, const Planes& Bp,
                  int64_t bn, int64_t bcols, int64_t br0, int64_t bc0, const Planes& Cp, int64_t cr0, int64_t cc0,
                  int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return B2M_OK;
    DOperand are{Ap.re, Ap.ld, an, an, ar0, ac0, true}, aim{Ap.im, Ap.ld, an, an, ar0, ac0, true};
    DOperand bre{Bp.re, Bp.ld, bn, bcols, br0, bc0, false}, bim{Bp.im, Bp.ld, bn, bcols, br0, bc0, false};
    double* cre = Cp.re + cr0 * Cp.ld + cc0;
    double* cim = Cp.im + cr0 * Cp.ld + cc0;
    B2M_TRY(dgemm_tiled(ctx, st, are, bre, cre, Cp.ld, M, N, K, B2M_DO_SUB, true));
    B2M_TRY(dgemm_tiled(ctx, st, aim, bim, cre, Cp.ld, M, N, K, B2M_DO_ADD, true));
    B2M_TRY(dgemm_tiled(ctx, st, are, bim, cim, Cp.ld, M, N, K, B2M_DO_SUB, true));
    return dgemm_tiled(ctx, st, aim, bre, cim, Cp.ld, M, N, K, B2M_DO_SUB, true);
}

int32_t launch_zstrip(Ctx* ctx, cudaStream_t st, ZStrip z, int splits, bool upper) {
    z.nsolve = (int)ceil_div(std::max(0, z.xhi - z.xlo), kZsCols);
    z.nleft = (int)ceil_div(z.left, kZsCols);
    z.nright = (int)ceil_div(std::max(0, z.end - z.right), kZsCols);
    z.status = ctx->d_status;
    const dim3 grid(z.nsolve + z.nleft + z.nright + (z.map && z.perm ? 1 : 0), splits);
    if (grid.x == 0) return B2M_OK;
    prof_begin(ctx, st, kClsTrsm);
    if (upper) zstrip_kernel<true><<<grid, kZsThreads, 0, st>>>(z);
    else zstrip_kernel<false><<<grid, kZsThreads, 0, st>>>(z);
    prof_end(ctx, st, kClsTrsm, 16.0 * (z.u1 - z.u0) * (2.0 * (z.xhi - z.xlo) + z.k));
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int64_t zsplit(int64_t w) { return round_up((w + 1) / 2, kZLeaf); }

// rows [br0, br0 + k) of X's columns [xc0, xc0 + ncols) <- T(r0..r0+k)^-1 X, T unit lower or upper
// (br0 = r0: the rows of X are T's)
int32_t ztrsm_rec(Ctx* ctx, cudaStream_t st, const Planes& T, int64_t tn, int64_t r0, const Planes& X, int64_t xn,
                  int64_t xcols, int64_t xc0, int64_t ncols, int64_t k, bool upper) {
    if (k <= kZBlock) {
        const int64_t nb = ceil_div(k, kZLeaf);
        for (int64_t i = 0; i < nb; ++i) {
            const int64_t b = (upper ? nb - 1 - i : i) * kZLeaf, kb = std::min<int64_t>(kZLeaf, k - b);
            ZStrip z{};
            z.T = T;
            z.X = X;
            z.r0 = (int)(r0 + b);
            z.k = (int)kb;
            z.u0 = (int)(upper ? r0 : r0 + b + kb);
            z.u1 = (int)(upper ? r0 + b : r0 + k);
            z.xlo = (int)xc0;
            z.xhi = (int)(xc0 + ncols);
            B2M_TRY(launch_zstrip(ctx, st, z, 1, upper));
        }
        return B2M_OK;
    }
    const int64_t k1 = zsplit(k), k2 = k - k1;
    if (!upper) {
        B2M_TRY(ztrsm_rec(ctx, st, T, tn, r0, X, xn, xcols, xc0, ncols, k1, false));
        B2M_TRY(zgemm_sub(ctx, st, T, tn, r0 + k1, r0, X, xn, xcols, r0, xc0, X, r0 + k1, xc0, k2, ncols, k1));
        return ztrsm_rec(ctx, st, T, tn, r0 + k1, X, xn, xcols, xc0, ncols, k2, false);
    }
    B2M_TRY(ztrsm_rec(ctx, st, T, tn, r0 + k1, X, xn, xcols, xc0, ncols, k2, true));
    B2M_TRY(zgemm_sub(ctx, st, T, tn, r0, r0 + k1, X, xn, xcols, r0 + k1, xc0, X, r0, xc0, k1, ncols, k2));
    return ztrsm_rec(ctx, st, T, tn, r0, X, xn, xcols, xc0, ncols, k1, true);
}

template <int RPT, bool MULTI>
int32_t launch_zpanel(Ctx* ctx, cudaStream_t st, const Planes& P, int m, int w, int row_base, int32_t* ipiv,
                      int32_t* map) {
    auto kern = zpanel_kernel<RPT, MULTI>;
    const int C = (int)ceil_div(m, RPT * kZNt), R = (int)ceil_div(m, C);
    std::atomic<int>& attr = device_flag((const void*)kern, 0, ctx->device);
    if (!attr.load()) {
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(RPT * kZNt * kZLeaf * sizeof(double2))));
        attr.store(1);
    }
    return launch_cluster(ctx, st, kern, !MULTI, C, kZNt, (size_t)R * kZLeaf * sizeof(double2), m, w, sizeof(double2), P, m, w,
                          R, row_base, ipiv, map, ctx->d_status, wait_polls(ctx));
}

// factor columns [c0, c0 + width), rows [c0, n); interchanges apply to all of [0, n)
int32_t zlu_rec(Ctx* ctx, cudaStream_t st, const Planes& A, int64_t n, int64_t c0, int64_t width, int32_t* ipiv,
                int32_t* perm, int32_t* map) {
    if (width <= kZBlock) {
        for (int64_t c = c0; c < c0 + width; c += kZLeaf) {
            const int w = (int)std::min<int64_t>(kZLeaf, c0 + width - c);
            const int64_t m = n - c;
            const Planes p{A.re + c * A.ld + c, A.im + c * A.ld + c, A.ld};
            ZStrip z{};
            z.T = z.X = A;
            z.r0 = (int)c;
            z.k = w;
            z.u0 = (int)(c + w);
            z.u1 = (int)n;
            z.xlo = (int)(c + w);
            z.xhi = (int)(c0 + width);
            // One row a thread while 8 CTAs hold the panel, then two; taller panels, whose rows 16 CTAs'
            // shared memory does not hold, on one CTA from L2.
            if (m <= kZMaxC * 2 * kZNt) {
                auto panel = m <= kZNt ? launch_zpanel<1, false>
                             : m <= 2 * kZNt ? launch_zpanel<2, false>
                             : m <= 8 * kZNt ? launch_zpanel<1, true> : launch_zpanel<2, true>;
                B2M_TRY(panel(ctx, st, p, (int)m, w, (int)c, ipiv, map));
                z.left = (int)c;
                z.right = (int)(c0 + width);
                z.end = (int)n;
                z.map = map;
                z.perm = perm;
            } else {
                prof_begin(ctx, st, kClsPanel);
                zpanel_tall_kernel<<<1, kZPanelThreads, 0, st>>>(p, (int)m, w, (int)c, (int)c, ipiv, ctx->d_status);
                prof_end(ctx, st, kClsPanel, 2.0 * 16.0 * m * w);
                B2M_LAUNCHED(ctx);
                B2M_TRY(launch_swaps<double>(ctx, st, A.re, A.ld, (int)n, (int)c, w, ipiv, perm));
                B2M_TRY(launch_swaps<double>(ctx, st, A.im, A.ld, (int)n, (int)c, w, ipiv, nullptr));
            }
            B2M_TRY(launch_zstrip(ctx, st, z, 1, false));
        }
        return B2M_OK;
    }
    const int64_t nleft = zsplit(width), nright = width - nleft, r1 = c0 + nleft;
    B2M_TRY(zlu_rec(ctx, st, A, n, c0, nleft, ipiv, perm, map));
    B2M_TRY(ztrsm_rec(ctx, st, A, n, c0, A, n, n, r1, nright, nleft, false));  // A12 <- L11^-1 A12
    B2M_TRY(zgemm_sub(ctx, st, A, n, r1, c0, A, n, n, c0, r1, A, r1, r1, n - r1, nright, nleft));
    return zlu_rec(ctx, st, A, n, r1, nright, ipiv, perm, map);
}

}  // namespace

int32_t zlu_factor(Ctx* ctx, cudaStream_t st, double* re, double* im, int64_t ld, int64_t n, int32_t* ipiv,
                   int32_t* perm) {
    if (n <= 0) return B2M_OK;
    if ((ld & 1) || !aligned16(re) || !aligned16(im)) return fail(ctx, B2M_ERR_DIM, "zlu_factor: alignment");
    if (n > (1 << 30)) return fail(ctx, B2M_ERR_UNSUPPORTED, "zlu_factor: n too large");
    const Planes A{re, im, ld};
    void* pm;
    B2M_TRY(ws_get(ctx, kWsPmap, (size_t)n * sizeof(int32_t), &pm));
    int32_t* map = static_cast<int32_t*>(pm);
    const GraphKey key{30, re, im, ipiv, perm, ld, n, 0, 0};
    return run_graph(ctx, st, key, [&](cudaStream_t s) -> int32_t {
        if (perm) {
            ziota_kernel<<<zblocks(n), 256, 0, s>>>(perm, n);
            B2M_LAUNCHED(ctx);
        }
        return zlu_rec(ctx, s, A, n, 0, n, ipiv, perm, map);
    });
}

int32_t zlu_solve(Ctx* ctx, cudaStream_t st, const double* lre, const double* lim, int64_t ld, int64_t n,
                  const int32_t* perm, double* bre, double* bim, int64_t ldb, int64_t nrhs, double* tre, double* tim) {
    if (n <= 0 || nrhs <= 0) return B2M_OK;
    const Planes L{const_cast<double*>(lre), const_cast<double*>(lim), ld};
    const Planes X{bre, bim, ldb}, W{tre, tim, ldb};
    // Steps of 32 rows out of place (so that several CTAs can share a strip's rows) while the right-hand sides
    // are few or the matrix is one block; else in place, split into GEMMs above kZBlock.  Kernels of a solve, steps
    // against GEMMs, ms: order 1100 64 right-hand sides 0.93 / 1.35, 256 1.03 / 1.39, 2048 2.06 / 1.88; order 2048
    // 1.85 / 3.48, 2.21 / 3.61, 5.66 / 4.83; order 3000 2.8 / 5.0, 3.6 / 5.2, 12.1 / 9.2.  The two meet between
    // 1000 and 2000 right-hand sides; from the line up to there the GEMMs cost up to 45 % more (order 2048, 512:
    // 2.7 / 3.9), and the line has not been moved.
    const bool steps = nrhs <= 256 || n <= kZBlock;
    const Planes& G = steps ? W : X;
    if (!steps) {
        B2M_CU(ctx, cudaMemcpy2DAsync(tre, ldb * 8, bre, ldb * 8, nrhs * 8, n, cudaMemcpyDeviceToDevice, st));
        B2M_CU(ctx, cudaMemcpy2DAsync(tim, ldb * 8, bim, ldb * 8, nrhs * 8, n, cudaMemcpyDeviceToDevice, st));
    }
    const Planes& S = steps ? X : W;
    zgather_rows_kernel<<<zblocks(n * nrhs), 256, 0, st>>>(G.re, G.im, ldb, S.re, S.im, ldb, perm, n, nrhs);
    B2M_LAUNCHED(ctx);
    if (!steps) {
        B2M_TRY(ztrsm_rec(ctx, st, L, n, 0, X, n, nrhs, 0, nrhs, n, false));
        return ztrsm_rec(ctx, st, L, n, 0, X, n, nrhs, 0, nrhs, n, true);
    }
    const int64_t nb = ceil_div(n, kZLeaf), strips = ceil_div(nrhs, kZsCols);
    for (int pass = 0; pass < 2; ++pass)
        for (int64_t i = 0; i < nb; ++i) {
            const int64_t b = (pass ? nb - 1 - i : i) * kZLeaf, kb = std::min<int64_t>(kZLeaf, n - b);
            ZStrip z{};
            z.T = L;
            z.X = pass ? X : W;
            z.Y = pass ? W : X;
            z.r0 = (int)b;
            z.k = (int)kb;
            z.u0 = (int)(pass ? 0 : b + kb);
            z.u1 = (int)(pass ? b : n);
            z.xhi = (int)nrhs;
            const int64_t splits = std::min<int64_t>(ceil_div(z.u1 - z.u0, 16 * kZsThreads / 32), 2 * ctx->num_sms / strips);
            B2M_TRY(launch_zstrip(ctx, st, z, (int)std::max<int64_t>(1, splits), pass != 0));
        }
    B2M_CU(ctx, cudaMemcpy2DAsync(bre, ldb * 8, tre, ldb * 8, nrhs * 8, n, cudaMemcpyDeviceToDevice, st));
    B2M_CU(ctx, cudaMemcpy2DAsync(bim, ldb * 8, tim, ldb * 8, nrhs * 8, n, cudaMemcpyDeviceToDevice, st));
    return B2M_OK;
}

int32_t z_deinterleave(Ctx* ctx, cudaStream_t st, const double* src, int64_t lws, double* re, double* im, int64_t ld,
                       int64_t rows, int64_t cols) {
    if (rows <= 0 || cols <= 0) return B2M_OK;
    deinterleave_kernel<<<zblocks(rows * cols), 256, 0, st>>>(src, lws, re, im, ld, rows, cols);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t z_interleave(Ctx* ctx, cudaStream_t st, double* dst, int64_t lwd, const double* re, const double* im,
                     int64_t ld, int64_t rows, int64_t cols, bool only_if_ok) {
    if (rows <= 0 || cols <= 0) return B2M_OK;
    interleave_kernel<<<zblocks(rows * cols), 256, 0, st>>>(dst, lwd, re, im, ld, rows, cols,
                                                            only_if_ok ? ctx->d_status : nullptr);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

int32_t z_determinant(Ctx* ctx, cudaStream_t st, const double* re, const double* im, int64_t ld, int64_t n,
                      const int32_t* ipiv, double* d_det2) {
    zdeterminant_kernel<<<1, 1024, 0, st>>>(Planes{const_cast<double*>(re), const_cast<double*>(im), ld}, (int)n,
                                            ipiv, ctx->d_status, d_det2);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

}  // namespace b2m
