// panel.cu -- partial-pivoting factorisation of one tall panel (the leaf of the LU recursion).
//
// panel_kernel factors leaves of up to 32 columns and 8192 rows; panel_push_kernel the narrower
// leaves (16 or 8 columns) of taller matrices, whose rows fill the shared memory of 16 CTAs.
//
// Pivot rule of the reference's leaf (LinAlgLU.pas:246-268), in both: largest |a|, lowest row among
// equals, singular when the largest |a| is <= 10/MaxDouble; the column below the pivot is scaled
// by the reciprocal 1/pivot (MatrixScaleAndAdd computes x*Scale + Offset with Offset = 0).
//
// panel_push_kernel: one thread-block cluster of C <= 16 CTAs factors an m x w panel (w <= W): CTA
// `rank` owns panel rows [rank*R, rank*R + R), thread t of a CTA owns rows t, t + 256, ...  Per
// column the CTAs exchange, by st.async pushes into every CTA's shared memory completing on that
// CTA's mbarrier, (a) their best pivot candidate with its full row and (b) the current diagonal row;
// each CTA then waits only on its own mbarrier and reads everything locally.  Receive buffers,
// warp-winner rows and the mbarriers are double buffered by column parity, which the causal order of
// the pushes makes race-free: a CTA pushes column j+1 only after it has finished reading everything
// of column j.
#include <cooperative_groups.h>

#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"
#include "panel.cuh"

namespace cg = cooperative_groups;

namespace b2m {
namespace {

constexpr int kPT = 256;              // threads per CTA
constexpr int kPWarps = kPT / 32;
constexpr int kPMaxC = 16;            // largest cluster
constexpr int kPanelSmemMax = 200 * 1024;  // dynamic shared memory a panel CTA may use

template <typename T> __device__ __forceinline__ T sing_thresh();
template <> __device__ __forceinline__ double sing_thresh<double>() { return 10.0 / DBL_MAX; }

// Warp argmax with the reference's tie rule, exactly: |a| >= 0 orders like its bit pattern, so
// the maximum is found with integer reductions (high word, then low word), and the lowest row
// index among the lanes holding it wins.  Lanes without a candidate carry (0, -1).
__device__ __forceinline__ void warp_best(double& a, int& i) {
    const unsigned long long b = i >= 0 ? (unsigned long long)__double_as_longlong(a) : 0ull;
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t mhi = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t m1 = __ballot_sync(0xffffffffu, hi == mhi && i >= 0);
    const uint32_t mlo = __reduce_max_sync(0xffffffffu, (m1 >> (threadIdx.x & 31)) & 1u ? lo : 0u);
    const bool top = i >= 0 && hi == mhi && lo == mlo;
    const uint32_t idx = __reduce_min_sync(0xffffffffu, top ? (uint32_t)i : 0xffffffffu);
    if (idx == 0xffffffffu) {
        a = 0.0;
        i = -1;
    } else {
        a = __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
        i = (int)idx;
    }
}
__device__ __forceinline__ uint4 pack_cand(double a, int i) {
    const unsigned long long b = __double_as_longlong(a);
    return make_uint4((uint32_t)b, (uint32_t)(b >> 32), (uint32_t)i, 0u);
}
__device__ __forceinline__ void unpack_cand(const uint32_t* w, double& a, int& i) {
    a = __longlong_as_double(((unsigned long long)w[1] << 32) | w[0]);
    i = (int)w[2];
}
__device__ __forceinline__ void st_async_b64(uint32_t raddr, unsigned long long v, uint32_t rbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n" ::"r"(raddr), "l"(v),
                 "r"(rbar)
                 : "memory");
}
__device__ __forceinline__ void st_async_elem(uint32_t raddr, double v, uint32_t rbar) {
    st_async_b64(raddr, (unsigned long long)__double_as_longlong(v), rbar);
}
// The panel lives in shared memory column-major (S[c*RS + local row], RS odd): a column is a
// contiguous, conflict-free vector, and a row is one element per lane.
template <typename T, int W, int RPT>
__global__ void __launch_bounds__(kPT, 1)
    panel_push_kernel(T* P, int64_t ld, int m, int w, int R, int row_base, int col_base, int32_t* ipiv,
                      int32_t* status, uint32_t polls) {
    constexpr int RB = W * (int)sizeof(T);  // row bytes

    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();

    extern __shared__ __align__(16) unsigned char panel_dyn[];
    T* S = reinterpret_cast<T*>(panel_dyn);
    const int RS = R | 1;

    __shared__ __align__(16) T rrow[2][kPMaxC][W];     // candidates' rows, by source CTA
    __shared__ __align__(16) T rdrow[2][W];            // the current diagonal row
    __shared__ __align__(16) uint32_t rcand[2][kPMaxC][4];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ T wabs[2][kPWarps];
    __shared__ int widx[2][kPWarps];
    __shared__ int s_late;  // a wait of the cluster ran out

    if (status[kInfo] != 0) return;  // uniform over the cluster: written before this launch

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lo = rank * R;
    const int hi = min(m, lo + R);
    const int nr = max(0, hi - lo);
    const uint32_t phase_bytes = (uint32_t)(C * (RB + 16) + RB);

    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        s_late = 0;
        fence_barrier_init();
    }
    // load this CTA's rows (row-major in global, column-major here), 16 loads in flight per thread
    {
        constexpr int B = 16;
        const int total = nr * W;
        for (int e0 = 0; e0 < total; e0 += B * kPT) {
            T v[B];
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const int e = e0 + q * kPT + tid;
                const int rl = e / W, c = e - rl * W;
                v[q] = (e < total && c < w) ? P[(int64_t)(lo + rl) * ld + c] : T(0);
            }
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const int e = e0 + q * kPT + tid;
                if (e < total) S[(e % W) * RS + e / W] = v[q];
            }
        }
    }
    cluster.sync();  // every mbarrier is initialised (and S is loaded) before the first push
    if (tid == 0) {
        mbar_arrive_expect_tx(&bar[0], phase_bytes);
        if (w > 1) mbar_arrive_expect_tx(&bar[1], phase_bytes);
    }

    // Columns are factored in blocks of BK: a block's columns live in registers (act), so each
    // column's scaling and rank-1 update touch registers only; the columns to the right of the
    // block receive one rank-BK update when the block is done.  Beyond the block, pushed rows are
    // therefore stale; the block's pivot rows get the missing triangular correction at the block
    // end (ublk), and every other row receives its own pending update with its own multipliers,
    // so each element sees exactly the sequence of rank-1 updates of the unblocked algorithm.
    constexpr int BK = 8;
    __shared__ __align__(16) T ublk[BK][W];
    int rowg[RPT];
    T act[RPT][BK];
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
        const int rl = tid + k * kPT;
        rowg[k] = rl < nr ? lo + rl : -1;
    }
    auto load_act = [&](const int jb) {
#pragma unroll
        for (int k = 0; k < RPT; ++k)
#pragma unroll
            for (int t = 0; t < BK; ++t)
                act[k][t] = (rowg[k] >= 0 && jb + t < W) ? S[(jb + t) * RS + tid + k * kPT] : T(0);
    };
    auto store_row = [&](const int k, const int jb) {
#pragma unroll
        for (int t = 0; t < BK; ++t)
            if (jb + t < w) S[(jb + t) * RS + tid + k * kPT] = act[k][t];
    };

    bool dead = false;  // this warp met a singular column or gave up a wait; the CTA leaves at its next barrier
    bool left = false;  // it has left
    // CTA-reduce the candidates of column `col` and push them, with the winner's row and the
    // diagonal row `col`, to every CTA of the cluster (block columns are taken from registers)
    auto publish = [&](const int col, T ma, int mi, const int jb) {
        const int par = col & 1;
        warp_best(ma, mi);
#pragma unroll
        for (int k = 0; k < RPT; ++k)
            if (rowg[k] >= 0 && ((mi >= 0 && rowg[k] == mi) || rowg[k] == col)) store_row(k, jb);
        if (lane == 0) { wabs[par][warp] = ma; widx[par][warp] = mi; }
        left = __syncthreads_or(dead);
        if (left) return;
        T a = lane < kPWarps ? wabs[par][lane] : T(0);
        int i = lane < kPWarps ? widx[par][lane] : -1;
        warp_best(a, i);
        const int wl = i >= 0 ? i - lo : 0;
        const bool own_diag = col >= lo && col < hi;
        for (int d = warp; d < C; d += kPWarps) {
            const uint32_t rb = map_rank(&bar[par], d);
            if (lane < W) {
                st_async_elem(map_rank(&rrow[par][rank][lane], d), S[lane * RS + wl], rb);
                if (own_diag) st_async_elem(map_rank(&rdrow[par][lane], d), S[lane * RS + (col - lo)], rb);
            }
            if (lane == 0) st_async16(map_rank(&rcand[par][rank][0], d), pack_cand(a, i), rb);
        }
        __syncthreads();  // rows read above are rewritten by the next column's interchange
    };

    load_act(0);
    {
        T ma = T(0);
        int mi = -1;
#pragma unroll
        for (int k = 0; k < RPT; ++k)
            if (rowg[k] >= 0 && fabs(act[k][0]) > ma) { ma = fabs(act[k][0]); mi = rowg[k]; }
        publish(0, ma, mi, 0);
    }
    int done = 0;  // columns whose pivot is recorded
    for (int jb = 0; jb < w && !dead && !left; jb += BK) {
#pragma unroll
        for (int t = 0; t < BK; ++t) {
            const int j = jb + t;
            if (j >= w) break;
            const int par = j & 1;
            const bool late = !cluster_wait(&bar[par], (j >> 1) & 1, polls, &s_late, C, status, 201);
            if (tid == 0 && !late && j + 2 < w) mbar_arrive_expect_tx(&bar[par], phase_bytes);
            // every warp derives the same pivot from the C candidates (lane c reads candidate c)
            T babs = T(0);
            int bidx = -1;
            if (lane < C) unpack_cand(&rcand[par][lane][0], babs, bidx);
            if (late) {  // above every candidate: the whole warp learns of it
                babs = static_cast<T>(__longlong_as_double(0x7ff8000000000000ll));
                bidx = 0x7fffffff;
            }
            warp_best(babs, bidx);
            if (bidx < 0 || !(babs > sing_thresh<T>())) {
                if (rank == 0 && tid == 0 && bidx != 0x7fffffff) atomicExch(&status[kInfo], 1);
                dead = true;
                break;
            }
            const int bc = bidx / R;  // the CTA that owns the pivot row sent its row
            const T* u = &rrow[par][bc][0];
            const T* dr = &rdrow[par][0];
            const int p = bidx;
            if (rank == 0 && tid == 0) ipiv[col_base + j] = row_base + p;
            done = j + 1;
            if (tid < W) ublk[t][tid] = u[tid];
            // the interchanged rows' columns outside the block: written lane-per-column by the
            // warp that owns each row (read only after the next barrier)
            if (j >= lo && j < hi && warp == ((j - lo) % kPT) >> 5 && lane < w && (lane < jb || lane >= jb + BK))
                S[lane * RS + (j - lo)] = u[lane];
            if (p != j && p >= lo && p < hi && warp == ((p - lo) % kPT) >> 5 && lane < w &&
                (lane < jb || lane >= jb + BK))
                S[lane * RS + (p - lo)] = dr[lane];
            const T rinv = T(1) / u[j];
            T mb = T(0);
            int mbi = -1;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int r = rowg[k];
                if (r < 0) continue;
                const int rl = tid + k * kPT;
                // interchange: row j takes the pivot row, row p the old diagonal row (block
                // columns in registers, the rest in shared memory, written by the row's owner)
                if (r == j || r == p) {
                    const T* src = r == j ? u : dr;
#pragma unroll
                    for (int t2 = 0; t2 < BK; ++t2) act[k][t2] = src[jb + t2];
                }
                if (r > j) {
                    const T l = act[k][t] * rinv + T(0);
                    act[k][t] = l;
#pragma unroll
                    for (int t2 = t + 1; t2 < BK; ++t2) act[k][t2] = fma(-l, u[jb + t2], act[k][t2]);
                    if (t + 1 < BK && fabs(act[k][t + 1]) > mb) { mb = fabs(act[k][t + 1]); mbi = r; }
                }
            }
            if (j + 1 >= w) continue;
            if (t + 1 < BK) {
                publish(j + 1, mb, mbi, jb);
                if (left) break;
                continue;
            }
            // ---- block end: correct the block's pivot rows beyond the block (L11^{-1} U12), store
            // the block columns, rank-BK update of the columns to the right, load the next block
            left = __syncthreads_or(false);
            if (left) break;
            for (int c = jb + BK + tid; c < w; c += kPT) {
#pragma unroll
                for (int t1 = 1; t1 < BK; ++t1) {
                    T x = ublk[t1][c];
#pragma unroll
                    for (int t0 = 0; t0 < t1; ++t0) x = fma(-ublk[t1][jb + t0], ublk[t0][c], x);
                    ublk[t1][c] = x;
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int r = rowg[k];
                if (r < 0) continue;
                const int rl = tid + k * kPT;
                store_row(k, jb);
                if (r > j) {
                    for (int c = jb + BK; c < w; ++c) {
                        T x = S[c * RS + rl];
#pragma unroll
                        for (int t2 = 0; t2 < BK; ++t2) x = fma(-act[k][t2], ublk[t2][c], x);
                        S[c * RS + rl] = x;
                    }
                } else if (r >= jb) {
                    for (int c = jb + BK; c < w; ++c) S[c * RS + rl] = ublk[r - jb][c];
                }
            }
            load_act(jb + BK);
            T ma = T(0);
            int mi = -1;
#pragma unroll
            for (int k = 0; k < RPT; ++k)
                if (rowg[k] > j && fabs(act[k][0]) > ma) { ma = fabs(act[k][0]); mi = rowg[k]; }
            publish(j + 1, ma, mi, jb + BK);
        }
    }
    if (!left) left = __syncthreads_or(dead);
    // (after a wait that ran out the rest of the leaf interchanges nothing: its readers find valid rows)
    if (left && rank == 0 && tid == 0 && *reinterpret_cast<volatile int*>(&s_late) != 0)
        for (int j = done; j < w; ++j) ipiv[col_base + j] = row_base + j;
    if (!left) {
        // the last block's columns are still in registers
        const int jl = ((w - 1) / BK) * BK;
#pragma unroll
        for (int k = 0; k < RPT; ++k)
            if (rowg[k] >= 0) store_row(k, jl);
    }
    __syncthreads();
    if (!left) {
        for (int e = tid; e < nr * w; e += kPT) {
            const int rl = e / w, c = e - rl * w;
            P[(int64_t)(lo + rl) * ld + c] = S[c * RS + rl];
        }
    }
    cluster_leave(&s_late);
}

template <typename T, int W, int RPT>
int32_t launch_push(Ctx* ctx, cudaStream_t st, int C, int R, T* P, int64_t ld, int m, int w, int row_base,
                    int col_base, int32_t* ipiv) {
    auto kern = panel_push_kernel<T, W, RPT>;
    const size_t smem = (size_t)W * (R | 1) * sizeof(T);
    std::atomic<int>& attr = device_flag((const void*)kern, 0, ctx->device);
    if (!attr.load()) {
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPanelSmemMax));
        attr.store(1);
    }
    return launch_cluster(ctx, st, kern, false, C, kPT, smem, m, w, sizeof(T), P, ld, m, w, R, row_base, col_base, ipiv,
                          ctx->d_status, wait_polls(ctx));
}


// ------------------------------------------------------------------------------------------
// panel_kernel: leaves of up to 32 columns and 8192 rows, on one CTA (up to 512 rows) or a cluster
// of up to 16.  What bounds a leaf is the chain of one column: find the largest |a| of all rows, get
// the pivot row to every row, update the next column.  A CTA is four main warps (one per scheduler)
// and a scribe warp; a thread owns RPT rows.  A CTA's rows live in shared memory; the eight columns
// of the current block also in registers, and every thread shifts its row left by one as a column is
// eliminated, so that the column loop is a compact body with compile-time register indices (the
// eight-times unrolled body of the first version missed in the instruction cache).  The chain is kept
// short by
//   * rows never moving: a thread carries its rows' current positions (the reference's interchanges
//     swap two positions), the diagonal row need not be sent, and rows go to their positions once,
//     at the end;
//   * deciding on the leading 32 bits of the magnitudes (one warp reduction and a ballot) and
//     comparing exactly, with the reference's first-maximum rule, only where those words tie;
//   * the reciprocal of each lane's best value running under the warp reduction;
//   * every warp sending its own candidate to all CTAs of the cluster (st.async on the receiver's
//     mbarrier; no CTA-level reduction first), and only the pieces its block can still use;
//   * the scribe warp recording pivots and the rows of U off the chain.
// At the end of a block of eight columns the pivot rows meet in every CTA (their multipliers and
// their columns right of the block), are solved with the block's L11 and update the other rows: each
// element sees the same products in the same order as without blocks, so the factors are bit for bit
// those of a column-by-column elimination.
// Measured on a B200 (32 columns, event-timed alone, before -> after): 100 rows 41.5 -> 21.2 us, 256
// rows 45.0 -> 22.5, 512 rows 54.0 -> 28.6, 1024 rows 53.3 -> 31.7, 2048 rows 53.2 -> 31.7, 4096 rows
// 55.3 -> 38.0, 8192 rows 56.4 -> 45.1 us (before: 256 threads, two barriers a column, pivot rows of
// 32 columns sent with every candidate).
// ------------------------------------------------------------------------------------------
constexpr int kPW = 32;              // columns
constexpr int kPNw = 4;              // main warps
constexpr int kPNt = kPNw * 32;      // main threads
constexpr int kPNa = kPNt + 32;      // with the scribe warp
constexpr int kPBk = 8;              // columns per block
// Candidates are kept for 16 columns: a CTA may push column j + 16 only after every CTA has sent
// column j + 15, and so has left the block of column j.
constexpr int kPSlots = 2 * kPBk;

// The previous leaf of the same outer panel (PanelLink::moves_in not null): the kernel first applies
// its interchanges, its triangular solve and its rank-32 update to the leaf's own columns, which still
// lack them.  As separate launches these were most of what lay between two leaves: 16 us for the
// interchanges with U12 (7,200 cycles of it composing the interchanges, which the scribe warp now
// does while the leaf is factored), 9 us for the update, and two launches.  In here they take 5.5 us
// (1024 and 2048 rows: 31.7 -> 37 us; 512 rows: 28.6 -> 37; 4096 rows: 38 -> 47).
// Moves: [0, 32) the row whose content ends in each of the leaf's rows, [32] the number of rows below
// the leaf that receive another row, [33, 65) these rows, [65, 97) the rows they receive.
constexpr int kPMoves = 3 * kPW + 1;
constexpr int kPLRows = 256;             // rows of L21 staged at a time
constexpr int kPLtPitch = kPW + 1;

// a warp's candidate for the pivot of a column
struct __align__(16) PCand {
    double rinv;       // 1 / row[0]
    int pos, lrow;     // position in the panel, local row of its CTA
    double row[kPBk];  // the row's block columns, from the current one on
};
static_assert(sizeof(PCand) == 80, "five 16-byte pieces");

// 16-byte pieces of a candidate of column `col` that the rest of its block can use
__device__ __forceinline__ int cand_pieces(int col) { return 1 + (kPBk + 1 - (col & (kPBk - 1))) / 2; }

template <int RPT, bool MULTI>
__global__ void __launch_bounds__(kPNa, 1)
    panel_kernel(double* P, int64_t ld, int m, int w, int R, int row_base, int col_base, int32_t* ipiv,
                 int32_t* status, PanelLink link, uint32_t polls) {
    int C = 1, rank = 0;
    if constexpr (MULTI) {
        C = (int)cg::this_cluster().num_blocks();
        rank = (int)cg::this_cluster().block_rank();
    }
    // this CTA's rows [R][kPW], the 16-byte pairs of a row swizzled so that a column read by 32 rows
    // and a row read by 16 lanes are both free of bank conflicts; after them (MULTI) s_rcv
    extern __shared__ __align__(16) double S[];
    auto sx = [](int row, int c) -> int { return row * kPW + 2 * ((c >> 1) ^ (row & 7)) + (c & 1); };
    __shared__ PCand s_loc[kPSlots][kPNw];  // candidates of this CTA's warps
    PCand (*s_rcv)[kPNw * kPMaxC] =         // candidates of the cluster's warps
        reinterpret_cast<PCand (*)[kPNw * kPMaxC]>(S + (size_t)kPW * R);
    __shared__ __align__(16) uint32_t s_key[2][kPNw];       // leading words of s_loc's values
    __shared__ __align__(16) double s_u[kPW][kPW];              // rows of U
    __shared__ __align__(16) double s_l[kPBk][kPBk];        // the block's rows of L11
    __shared__ __align__(8) uint64_t s_bar[kPSlots], s_rbar;    // a column's candidates; a block's pivot rows
    __shared__ int s_pl[kPW], s_ps[kPW];                        // the pivots: local row, CTA
    __shared__ int s_mv[kPMoves];
    __shared__ int s_late;    // a wait of the cluster ran out
    __shared__ PCand s_none;  // no candidate
    // Staging of the previous leaf's L21 rows (s_ll) and of its L11, then U12 (s_lt).  In a cluster it
    // lies in s_rcv: slot 0 may be written by CTAs that are done with their prologue, slots 1 .. 13
    // hold s_ll (no candidate of column 1 is sent before every CTA has sent column 0), the last two
    // s_lt (not written before the scribe has left column 7).
    double* s_ll = MULTI ? reinterpret_cast<double*>(&s_rcv[1][0]) : S + (size_t)kPW * R;
    double* s_lt = MULTI ? reinterpret_cast<double*>(&s_rcv[kPSlots - 2][0]) : s_ll + kPW * kPLRows;
    static_assert(sizeof(PCand) * kPNw * kPMaxC * (kPSlots - 3) >= sizeof(double) * kPW * kPLRows, "s_ll fits");
    static_assert(sizeof(PCand) * kPNw * kPMaxC * 2 >= sizeof(double) * kPW * kPLtPitch, "s_lt fits");
    if (status[kInfo] != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lo = rank * R;
    const int nr = max(0, min(m, lo + R) - lo);
    if constexpr (MULTI) {
        // every CTA's barriers are initialised before the first push; the wait comes after the loads
        // One barrier per candidate slot: the scribe may be up to a block of columns behind the main
        // warps, and must not miss a phase (with two barriers, two columns on, it would wait for one
        // that has passed).
        if (tid == 0) {
            for (int j = 0; j < kPSlots; ++j) mbar_init(&s_bar[j], 1);
            mbar_init(&s_rbar, 1);
            s_late = 0;
            s_none.row[0] = 0.0;
            fence_barrier_init();
            for (int j = 0; j < min(kPSlots, w); ++j)
                mbar_arrive_expect_tx(&s_bar[j], (uint32_t)(C * kPNw * 16 * cand_pieces(j)));
            mbar_arrive_expect_tx(&s_rbar, (uint32_t)(min(kPBk, w) * kPW * 8));
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    }
    const bool linked = link.moves_in != nullptr;
    {
        constexpr int RS = kPNa / (kPW / 2);  // rows per step
        const int c = 2 * (tid % (kPW / 2));
        const int bytes = c + 1 < w ? 16 : (c < w ? 8 : 0), cc = c < w ? c : 0;
        if (!linked) {
            const double* src = P + (int64_t)(lo + tid / (kPW / 2)) * ld + cc;
#pragma unroll 4
            for (int rl = tid / (kPW / 2); rl < nr; rl += RS, src += RS * ld) cp_async16(S + sx(rl, c), src, bytes);
            cp_async_commit();
        } else {
            // the rows as the previous leaf's interchanges leave them, its top rows (positions -32 .. -1
            // here) and its L11 first, then this CTA's rows and their multipliers
            int* s_map = reinterpret_cast<int*>(&s_loc[0][0]);
            static_assert(sizeof(s_loc) >= (size_t)kPNt * RPT * sizeof(int), "the row map fits");
            const int mv = tid < kPMoves ? link.moves_in[tid] : 0;  // (fewer moves than threads)
            for (int rl = tid; rl < nr; rl += kPNa) s_map[rl] = lo + rl;
            if (tid < kPMoves) s_mv[tid] = mv;
            __syncthreads();
            if (tid < s_mv[kPW]) {
                const int d = s_mv[kPW + 1 + tid] - row_base - lo;
                if (d >= 0 && d < nr) s_map[d] = s_mv[2 * kPW + 1 + tid] - row_base;
            }
            for (int rl = tid / (kPW / 2); rl < kPW; rl += RS)
                cp_async16(&s_u[rl][c], P + (int64_t)(s_mv[rl] - row_base) * ld + cc, bytes);
            for (int e = tid; e < kPW * kPW; e += kPNa)
                cp_async8(s_lt + (e >> 5) * kPLtPitch + (e & 31), P + (int64_t)((e >> 5) - kPW) * ld + (e & 31) - kPW, 8);
            cp_async_commit();
            __syncthreads();
#pragma unroll 4
            for (int rl = tid / (kPW / 2); rl < nr; rl += RS)
                cp_async16(S + sx(rl, c), P + (int64_t)s_map[rl] * ld + cc, bytes);
            const double* src = P + (int64_t)(lo + tid / (kPW / 2)) * ld + c - kPW;
#pragma unroll 4
            for (int rl = tid / (kPW / 2); rl < min(nr, kPLRows); rl += RS, src += RS * ld)
                cp_async16(s_ll + sx(rl, c), src, 16);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            if (warp < kPNw) {
                // U12 = L11^-1 (top rows): warp = 8 columns, lane = column + 8 * (row & 3); four rows a
                // step, the finished element broadcast by a shuffle; contributions in ascending order
                const int col = 8 * warp + (lane & 7), rg = lane >> 3;
                double x[kPW / 4];
#pragma unroll
                for (int i = 0; i < kPW / 4; ++i) x[i] = s_u[4 * i + rg][col];
#pragma unroll 1
                for (int q = 0; q < kPW / 4; ++q) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const double xi = __shfl_sync(0xffffffffu, x[0], (lane & 7) + 8 * t);
                        const double* lt = s_lt + (4 * q + rg) * kPLtPitch + 4 * q + t;
                        if (rg > t) x[0] = fma(-lt[0], xi, x[0]);
#pragma unroll
                        for (int i = 1; i < kPW / 4; ++i)
                            if (q + i < kPW / 4) x[i] = fma(-lt[4 * i * kPLtPitch], xi, x[i]);
                    }
                    s_u[4 * q + rg][col] = x[0];
#pragma unroll
                    for (int i = 1; i < kPW / 4; ++i) x[i - 1] = x[i];
                }
            }
            cp_async_wait<0>();
            __syncthreads();
            // rows -= L21 U12 on the FP64 tensor cores, 16 rows a step; U12's fragments stay in registers
            // (a = L21[g][k + t], L21[g + 8][k + t], b = U12[k + t][g], c = rows g, g + 8, columns 2t, 2t + 1)
            if (warp < kPNw) {
                const int g = lane >> 2, t = lane & 3;
                double bf[kPW / 4][kPW / 8];
#pragma unroll
                for (int k = 0; k < kPW / 4; ++k)
#pragma unroll
                    for (int j = 0; j < kPW / 8; ++j) bf[k][j] = s_u[4 * k + t][8 * j + g];
                for (int ch = 0; ch < nr; ch += kPLRows) {
                    if (ch > 0) {  // the next rows' multipliers take the place of the last ones
                        asm volatile("bar.sync 3, %0;\n" ::"n"(kPNt) : "memory");
                        constexpr int RM = kPNt / (kPW / 2);
#pragma unroll 4
                        for (int rl = ch + tid / (kPW / 2); rl < min(nr, ch + kPLRows); rl += RM)
                            cp_async16(s_ll + sx(rl - ch, c), P + (int64_t)(lo + rl) * ld + c - kPW, 16);
                        cp_async_commit();
                        cp_async_wait<0>();
                        asm volatile("bar.sync 3, %0;\n" ::"n"(kPNt) : "memory");
                    }
#pragma unroll 1
                    for (int r0 = ch + 16 * warp; r0 < min(nr, ch + kPLRows); r0 += 16 * kPNw) {
                        const int ra = r0 + g, rb = ra + 8;
                        const bool oka = ra < nr, okb = rb < nr;
                        double acc[kPW / 8][4] = {};
#pragma unroll
                        for (int k = 0; k < kPW / 4; ++k) {
                            const double a0 = oka ? s_ll[sx(ra - ch, 4 * k + t)] : 0.0;
                            const double a1 = okb ? s_ll[sx(rb - ch, 4 * k + t)] : 0.0;
#pragma unroll
                            for (int j = 0; j < kPW / 8; ++j)
                                asm volatile(
                                    "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
                                    "{%0,%1,%2,%3};\n"
                                    : "+d"(acc[j][0]), "+d"(acc[j][1]), "+d"(acc[j][2]), "+d"(acc[j][3])
                                    : "d"(a0), "d"(a1), "d"(bf[k][j]));
                        }
#pragma unroll
                        for (int j = 0; j < kPW / 8; ++j) {
                            double2* pa = reinterpret_cast<double2*>(S + sx(ra, 8 * j + 2 * t));
                            double2* pb = reinterpret_cast<double2*>(S + sx(rb, 8 * j + 2 * t));
                            if (oka) *pa = make_double2(pa->x - acc[j][0], pa->y - acc[j][1]);
                            if (okb) *pb = make_double2(pb->x - acc[j][2], pb->y - acc[j][3]);
                        }
                    }
                }
                // U12 out of the way of this leaf's U (L11 is no longer read)
                for (int e = tid; e < kPW * kPW; e += kPNt) s_lt[(e >> 5) * kPLtPitch + (e & 31)] = s_u[e >> 5][e & 31];
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    if constexpr (MULTI) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    bool late = false;  // this thread, after select() some thread of its warp, gave up a wait (see panel.cuh)
    // the pivot of column j among the published candidates, the same in every warp (none for a warp that is late)
    auto select = [&](const int j, int& win) -> const PCand* {
        const int slot = j & (kPSlots - 1);
        if constexpr (MULTI) {
            const PCand* cands = s_rcv[slot];
            const int cnt = C * kPNw;
            uint32_t k[2], mk = 0;
            int q = lane;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                k[e] = lane + 32 * e < cnt ? mag_hi(cands[lane + 32 * e].row[0]) : 0u;
                mk = max(mk, k[e]);
            }
            int n = 0;
#pragma unroll
            for (int e = 1; e >= 0; --e) {
                n += k[e] == mk ? 1 : 0;
                q = k[e] == mk ? lane + 32 * e : q;
            }
            const uint32_t M = __reduce_max_sync(0xffffffffu, mk);
            const uint32_t bal = __ballot_sync(0xffffffffu, mk == M);
            const uint32_t bal2 = __ballot_sync(0xffffffffu, late || (mk == M && n > 1));
            int wl = __ffs(bal) - 1;
            if ((bal & (bal - 1)) || bal2) {
                late = __any_sync(0xffffffffu, late);
                if (late) {
                    win = 0;
                    return &s_none;
                }
                double ba = 0.0;
                int bp = 0x7fffffff;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (lane + 32 * e >= cnt) continue;
                    const double a = fabs(cands[lane + 32 * e].row[0]);
                    const int p = cands[lane + 32 * e].pos;
                    if (a > ba || (a == ba && p < bp)) { ba = a; bp = p; q = lane + 32 * e; }
                }
                wl = warp_winner(ba, bp);
            }
            const uint32_t odd = __ballot_sync(0xffffffffu, q >= 32);
            win = wl + (((odd >> wl) & 1u) ? 32 : 0);
            if (win >= cnt) win = 0;
            return &cands[win];
        } else {
            const uint4 kv = *reinterpret_cast<const uint4*>(&s_key[j & 1][0]);
            const uint32_t k[kPNw] = {kv.x, kv.y, kv.z, kv.w};
            const uint32_t M = max(max(k[0], k[1]), max(k[2], k[3]));
            int n = 0;
            win = 0;
#pragma unroll
            for (int q = kPNw - 1; q >= 0; --q) {
                win = k[q] == M ? q : win;
                n += k[q] == M ? 1 : 0;
            }
            if (n > 1) {
                const PCand* cands = s_loc[slot];
                win = warp_winner(lane < kPNw ? fabs(cands[lane].row[0]) : 0.0,
                                  lane < kPNw ? cands[lane].pos : 0x7fffffff);
                if (win >= kPNw) win = 0;
            }
            return &s_loc[slot][win];
        }
    };
    auto wait_bar = [&](uint64_t* bar, const uint32_t phase, const int site) {
        late = !cluster_wait(bar, phase, polls, &s_late, C, status, site);
    };
    auto wait_col = [&](const int j) { wait_bar(&s_bar[j & (kPSlots - 1)], j / kPSlots, 201); };
    bool dead = false;  // this warp met a singular column or is late; the CTA leaves at the next barrier 2
    bool left = false;  // it has left
    if (warp == kPNw) {
        // ---- scribe warp: records each pivot, and the pivot row's part of U inside its block
        // It also composes the interchanges into moves: lane i holds the position whose content ends in
        // position i (sm), lane e < n_extra a position below the leaf that an interchange reached and
        // the one whose content ends there.
        int sm = lane, my_pos = -1, my_src = -1, n_extra = 0, j = 0;
        for (int jb = 0; jb < w && !left; jb += kPBk) {
            for (; j < min(jb + kPBk, w); ++j) {
                if constexpr (MULTI) {
                    wait_col(j);
                } else {
                    asm volatile("bar.sync 1, %0;\n" ::"r"(kPNa) : "memory");
                }
                int win;
                const PCand* b = select(j, win);
                const double v = lane < kPBk ? b->row[lane] : 0.0;
                if (!(fabs(b->row[0]) > sing_thresh<double>())) {
                    dead = true;
                    break;
                }
                if (j == 0 && linked && rank == 0) {
                    // every CTA has read its rows: U12 of the previous leaf takes its place
#pragma unroll 8
                    for (int r = 0; r < kPW; ++r)
                        if (lane < w) P[(int64_t)(r - kPW) * ld + lane] = s_lt[r * kPLtPitch + lane];
                }
                {
                    const int q = b->pos, a = __shfl_sync(0xffffffffu, sm, j);
                    int other;
                    if (q < w) {
                        other = __shfl_sync(0xffffffffu, sm, q);
                        if (lane == q) sm = a;
                    } else {
                        const uint32_t hit = __ballot_sync(0xffffffffu, my_pos == q);
                        const int e = hit ? __ffs(hit) - 1 : n_extra++;
                        if (!hit && lane == e) my_pos = my_src = q;
                        other = __shfl_sync(0xffffffffu, my_src, e);
                        if (lane == e) my_src = a;
                    }
                    if (lane == j) sm = other;
                }
                if (lane < kPBk && (j & (kPBk - 1)) + lane < kPBk && j + lane < kPW) s_u[j][j + lane] = v;
                if (lane == 0) {
                    if (rank == 0) ipiv[col_base + j] = row_base + b->pos;
                    s_pl[j] = b->lrow;
                    s_ps[j] = MULTI ? win / kPNw : 0;
                }
            }
            left = bar_any<kPNa>(2, dead);
            if (jb + kPBk < w && !left) left = bar_any<kPNa>(2, false);
        }
        const bool gave_up = MULTI && left && *reinterpret_cast<volatile int*>(&s_late) != 0;
        // after a wait that ran out the rest of the leaf interchanges nothing: its readers find valid rows
        if (gave_up && rank == 0 && lane >= j && lane < w) ipiv[col_base + lane] = row_base + lane;
        if ((!left || gave_up) && rank == 0 && link.moves_out) {
            link.moves_out[lane] = row_base + sm;
            if (lane == 0) link.moves_out[kPW] = n_extra;
            link.moves_out[kPW + 1 + lane] = row_base + my_pos;
            link.moves_out[2 * kPW + 1 + lane] = row_base + my_src;
        }
    } else {
        int pos[RPT];
        double act[RPT][kPBk];
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int rl = tid + r * kPNt;
            pos[r] = rl < nr ? lo + rl : -1 - kPW;
#pragma unroll
            for (int i = 0; i < kPBk; i += 2) {
                const double2 x =
                    rl < nr ? *reinterpret_cast<const double2*>(S + sx(rl, i)) : make_double2(0.0, 0.0);
                act[r][i] = x.x; act[r][i + 1] = x.y;
            }
        }
        // lane l sends to CTA l & 15 of the cluster, pieces (l >> 4), (l >> 4) + 2, ...
        uint32_t push_dst = 0, push_bar = 0;
        if constexpr (MULTI) {
            const int d = min(lane & 15, C - 1);
            push_dst = map_rank(&s_rcv[0][rank * kPNw + warp], d);
            push_bar = map_rank(&s_bar[0], d);
        }
        // the warp's best candidate of the column held in act[.][0]: the leading words decide (an
        // exact comparison only where they tie or are not finite); every lane prepares its own best
        // row's reciprocal meanwhile
        auto publish = [&](const int col) {
            const int slot = col & (kPSlots - 1);
            uint32_t h[RPT], mh = 0;
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                h[r] = pos[r] >= 0 ? mag_hi(act[r][0]) : 0u;
                mh = max(mh, h[r]);
            }
            double cr[kPBk];
            int cp = pos[0], cl = tid, cnt = h[0] == mh ? 1 : 0;
#pragma unroll
            for (int i = 0; i < kPBk; ++i) cr[i] = act[0][i];
#pragma unroll
            for (int r = 1; r < RPT; ++r) {
                const bool is = h[r] == mh;
                cnt += is ? 1 : 0;
#pragma unroll
                for (int i = 0; i < kPBk; ++i) cr[i] = is ? act[r][i] : cr[i];
                cp = is ? pos[r] : cp;
                cl = is ? tid + r * kPNt : cl;
            }
            cr[0] = mh != 0 ? cr[0] : 0.0;
            // (the select is opaque: the compiler would otherwise divide 1 by a candidate-less lane's
            // zero, whose slow path costs the whole warp ~170 cycles)
            double rarg;
            asm("{ .reg .pred p; setp.ne.u32 p, %2, 0; selp.f64 %0, %1, 0d3FF0000000000000, p; }"
                : "=d"(rarg)
                : "d"(cr[0]), "r"(mh));
            double rinv = 1.0 / rarg;
            const uint32_t M = __reduce_max_sync(0xffffffffu, mh);
            const uint32_t b1 = __ballot_sync(0xffffffffu, mh == M);
            const uint32_t b2 = __ballot_sync(0xffffffffu, mh == M && cnt > 1);
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
                        cl = tid + r * kPNt;
#pragma unroll
                        for (int i = 0; i < kPBk; ++i) cr[i] = act[r][i];
                    }
                }
                if (!(ba > 0.0)) cr[0] = 0.0;
                rinv = 1.0 / (ba > 0.0 ? cr[0] : 1.0);
                wl = warp_winner(ba, cp);
            }
            if (lane == wl) {
                PCand& c = s_loc[slot][warp];
#pragma unroll
                for (int i = 0; i < kPBk; i += 2)
                    *reinterpret_cast<double2*>(&c.row[i]) = make_double2(cr[i], cr[i + 1]);
                c.rinv = rinv;
                *reinterpret_cast<int2*>(&c.pos) = make_int2(M != 0 ? cp : 0x7fffffff, cl);
                if (!MULTI) s_key[col & 1][warp] = mag_hi(cr[0]);
            }
            if constexpr (MULTI) {
                __syncwarp();
                const uint4* src = reinterpret_cast<const uint4*>(&s_loc[slot][warp]);
                const int np = cand_pieces(col);
                const uint32_t rdst = push_dst + slot * (uint32_t)(kPNw * kPMaxC * sizeof(PCand));
                const uint32_t rbar = push_bar + 8 * slot;
                if ((lane & 15) < C)
                    for (int q = lane >> 4; q < np; q += 2) st_async16(rdst + 16 * q, src[q], rbar);
            }
        };
        publish(0);
        for (int jb = 0; jb < w; jb += kPBk) {
            const int bw = min(kPBk, w - jb);
#pragma unroll 1
            for (int t = 0; t < bw; ++t) {
                const int j = jb + t;
                if constexpr (MULTI) {
                    wait_col(j);
                    if (tid == 0 && !late && j + kPSlots < w)
                        mbar_arrive_expect_tx(&s_bar[j & (kPSlots - 1)],
                                              (uint32_t)(C * kPNw * 16 * cand_pieces(j + kPSlots)));
                } else {
                    asm volatile("bar.sync 1, %0;\n" ::"r"(kPNa) : "memory");
                }
                int win;
                const PCand* b = select(j, win);
                double u[kPBk];
#pragma unroll
                for (int i = 0; i < kPBk; i += 2) {
                    const double2 x = *reinterpret_cast<const double2*>(&b->row[i]);
                    u[i] = x.x; u[i + 1] = x.y;
                }
                const double rinv = b->rinv;
                const int2 pl = *reinterpret_cast<const int2*>(&b->pos);
                const int p = pl.x, lrow = pl.y;
                if (!(fabs(u[0]) > sing_thresh<double>())) {
                    if (rank == 0 && tid == 0 && !late) atomicExch(&status[kInfo], 1);
                    dead = true;
                    break;
                }
                const bool mine = MULTI ? win / kPNw == rank : true;
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    const int rl = tid + r * kPNt;
                    if (mine && rl == lrow) pos[r] = -1 - j;
                    else if (pos[r] == j) pos[r] = p;
                    const double l = act[r][0] * rinv + 0.0;
                    if (pos[r] >= 0) S[sx(rl, j)] = l;
#pragma unroll
                    for (int i = 1; i < kPBk; ++i) act[r][i - 1] = fma(-l, u[i], act[r][i]);
                    act[r][kPBk - 1] = 0.0;
                }
                if (t + 1 < bw) publish(j + 1);
            }
            // ---- block end: the pivot rows as their owners hold them (multipliers, and the columns
            // right of the block without the block's updates) come together in every CTA
            const int c1 = jb + kPBk;
            if (c1 >= w) break;
            left = bar_any<kPNa>(2, dead);
            if (left) break;
            if constexpr (MULTI) {
                for (int e = tid; e < kPBk * (kPW / 2); e += kPNt) {
                    const int t = e / (kPW / 2), q = e - t * (kPW / 2), c = 2 * q;
                    if (s_ps[jb + t] == rank && (c >= c1 || (c >= jb && c < jb + kPBk))) {
                        const double2 x = *reinterpret_cast<const double2*>(S + sx(s_pl[jb + t], c));
                        const unsigned long long xb = __double_as_longlong(x.x), yb = __double_as_longlong(x.y);
                        const uint4 xv =
                            make_uint4((uint32_t)xb, (uint32_t)(xb >> 32), (uint32_t)yb, (uint32_t)(yb >> 32));
                        double* dst = c >= c1 ? &s_u[jb + t][c] : &s_l[t][c - jb];
                        for (int d = 0; d < C; ++d) st_async16(map_rank(dst, d), xv, map_rank(&s_rbar, d));
                    }
                }
                wait_bar(&s_rbar, (jb / kPBk) & 1, 203);
            } else {
                for (int e = tid; e < kPBk * (kPW / 2); e += kPNt) {
                    const int t = e / (kPW / 2), q = e - t * (kPW / 2), c = 2 * q;
                    const double2 x = *reinterpret_cast<const double2*>(S + sx(s_pl[jb + t], c));
                    if (c >= c1) *reinterpret_cast<double2*>(&s_u[jb + t][c]) = x;
                    else if (c >= jb) *reinterpret_cast<double2*>(&s_l[t][c - jb]) = x;
                }
                asm volatile("bar.sync 3, %0;\n" ::"r"(kPNt) : "memory");
            }
            if (warp == 0 && c1 + lane < kPW) {
                // U right of the block: L11^-1 times the rows, contributions in ascending order
                const int c = c1 + lane;
                double x[kPBk];
#pragma unroll
                for (int q = 0; q < kPBk; ++q) x[q] = s_u[jb + q][c];
#pragma unroll
                for (int t0 = 0; t0 < kPBk - 1; ++t0)
#pragma unroll
                    for (int t1 = t0 + 1; t1 < kPBk; ++t1) x[t1] = fma(-s_l[t1][t0], x[t0], x[t1]);
#pragma unroll
                for (int q = 1; q < kPBk; ++q) s_u[jb + q][c] = x[q];
            }
            if (MULTI && tid == 0 && !late)
                mbar_arrive_expect_tx(&s_rbar, (uint32_t)(min(kPBk, w - c1) * (kPW - c1) * 8));
            double l[RPT][kPBk];
#pragma unroll
            for (int r = 0; r < RPT; ++r)
#pragma unroll
                for (int q = 0; q < kPBk; q += 2) {
                    const int rl = tid + r * kPNt;
                    double2 x = make_double2(0.0, 0.0), y = x;
                    if (pos[r] >= 0) {
                        x = *reinterpret_cast<const double2*>(S + sx(rl, jb + q));
                        y = *reinterpret_cast<const double2*>(S + sx(rl, c1 + q));
                    }
                    l[r][q] = x.x; l[r][q + 1] = x.y;
                    act[r][q] = y.x; act[r][q + 1] = y.y;
                }
            left = bar_any<kPNa>(2, late);
            if (left) break;
#pragma unroll
            for (int i = 0; i < kPBk; i += 2)
#pragma unroll
                for (int q = 0; q < kPBk; ++q) {
                    const double2 uu = *reinterpret_cast<const double2*>(&s_u[jb + q][c1 + i]);
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        act[r][i] = fma(-l[r][q], uu.x, act[r][i]);
                        act[r][i + 1] = fma(-l[r][q], uu.y, act[r][i + 1]);
                    }
                }
            publish(c1);
#pragma unroll 1
            for (int c = c1 + kPBk; c < w; c += 2) {
                double2 x[RPT];
#pragma unroll
                for (int r = 0; r < RPT; ++r)
                    x[r] = pos[r] >= 0 ? *reinterpret_cast<const double2*>(S + sx(tid + r * kPNt, c))
                                       : make_double2(0.0, 0.0);
#pragma unroll
                for (int q = 0; q < kPBk; ++q) {
                    const double2 uu = *reinterpret_cast<const double2*>(&s_u[jb + q][c]);
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        x[r].x = fma(-l[r][q], uu.x, x[r].x);
                        x[r].y = fma(-l[r][q], uu.y, x[r].y);
                    }
                }
#pragma unroll
                for (int r = 0; r < RPT; ++r)
                    if (pos[r] >= 0) *reinterpret_cast<double2*>(S + sx(tid + r * kPNt, c)) = x[r];
            }
        }
        if (!left) left = bar_any<kPNa>(2, dead);
        if (!left) {
            // every row goes to its position: rows below the pivots as they are (multipliers), the
            // pivot rows held here with U right of the diagonal
            int* s_pos = reinterpret_cast<int*>(&s_loc[0][0]);
            static_assert(sizeof(s_loc) >= (size_t)kPNt * RPT * sizeof(int), "positions fit");
#pragma unroll
            for (int r = 0; r < RPT; ++r) s_pos[tid + r * kPNt] = pos[r];
            asm volatile("bar.sync 3, %0;\n" ::"r"(kPNt) : "memory");
            constexpr int LPR = kPW / 2;    // lanes per row, two columns a lane
            constexpr int RS = kPNt / LPR;  // rows per step
            constexpr int BP = kPW / RS < 4 ? kPW / RS : 4, B = 8;
            const int c = 2 * (tid % LPR);
            auto put = [&](int row, double2 x) {
                if (row >= m) return;
                double* dst = P + (int64_t)row * ld + c;
                if (c + 1 < w) *reinterpret_cast<double2*>(dst) = x;
                else if (c < w) *dst = x.x;
            };
            for (int j0 = tid / LPR; j0 < w; j0 += RS * BP) {
                double2 x[BP], u[BP];
                bool mine[BP];
#pragma unroll
                for (int b = 0; b < BP; ++b) {
                    const int j = min(j0 + b * RS, w - 1);
                    mine[b] = s_ps[j] == rank && j0 + b * RS < w;
                    x[b] = *reinterpret_cast<const double2*>(S + sx(mine[b] ? s_pl[j] : 0, c));
                    u[b] = *reinterpret_cast<const double2*>(&s_u[j][c]);
                }
#pragma unroll
                for (int b = 0; b < BP; ++b) {
                    const int j = j0 + b * RS;
                    if (mine[b]) put(j, make_double2(c >= j ? u[b].x : x[b].x, c + 1 >= j ? u[b].y : x[b].y));
                }
            }
            for (int r0 = tid / LPR; r0 < nr; r0 += RS * B) {
                double2 x[B];
                int q[B];
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    const int rl = min(r0 + b * RS, nr - 1);
                    q[b] = r0 + b * RS < nr ? s_pos[rl] : -1;
                    x[b] = *reinterpret_cast<const double2*>(S + sx(rl, c));
                }
#pragma unroll
                for (int b = 0; b < B; ++b)
                    if (q[b] >= 0) put(q[b], x[b]);
            }
        }
    }
    if constexpr (MULTI) cluster_leave(&s_late);
}

template <int RPT, bool MULTI>
int32_t launch_panel32(Ctx* ctx, cudaStream_t st, int C, double* P, int64_t ld, int m, int w, int row_base,
                       int col_base, int32_t* ipiv, const PanelLink& link) {
    auto kern = panel_kernel<RPT, MULTI>;
    const int R = (int)ceil_div(m, C);
    constexpr size_t staged = (kPW * kPLRows + kPW * kPLtPitch) * sizeof(double);
    constexpr size_t extra = MULTI ? sizeof(PCand) * kPSlots * kPNw * kPMaxC : staged;
    const size_t smem = (size_t)kPW * R * sizeof(double) + (MULTI || link.moves_in ? extra : 0);
    std::atomic<int>& attr = device_flag((const void*)kern, 0, ctx->device);
    if (!attr.load()) {
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kPW * kPNt * RPT * sizeof(double) + extra)));
        attr.store(1);
    }
    return launch_cluster(ctx, st, kern, !MULTI, C, kPNa, smem, m, w, sizeof(double), P, ld, m, w, R, row_base, col_base,
                          ipiv, ctx->d_status, link, wait_polls(ctx));
}

}  // namespace

// Tallest panel of width w: 16 CTAs of 512 rows (w <= 32), 1024 (w <= 16) or 2048 (w <= 8), by what the
// shared memory of a CTA holds.
int panel_max_rows(bool fp64, int w) {
    if (fp64) return w <= 8 ? kPMaxC * kPT * 8 : (w <= 16 ? kPMaxC * kPT * 4 : kPMaxC * kPT * 2);
    return kPMaxC * kPT * 4;
}

template <typename T>
int32_t launch_panel(Ctx* ctx, cudaStream_t st, T* P, int64_t ld, int m, int w, int row_base, int col_base,
                     int32_t* ipiv, const PanelLink& link) {
    if (w < 1 || w > 32 || m < w) return fail(ctx, B2M_ERR_DIM, "panel %d x %d", m, w);
    if constexpr (sizeof(T) == 8) {
        // Rows per thread (measured, 32 columns): up to 512 rows one CTA, 22.5 us at 256 rows with two
        // rows a thread (28.6 us at 512 with four; a cluster of two took 30.7); above, two rows a
        // thread while 8 CTAs hold the panel (31.7 us at 1024 and 2048 rows; four: 37.8), then four,
        // which needs half the CTAs (38.0 us at 4096 rows; 38.9 on 16 CTAs).
        if (m <= kPMaxC * kPNt * 4 && aligned16(P) && ld % 2 == 0) {
            if (m <= 2 * kPNt)
                return launch_panel32<2, false>(ctx, st, 1, P, ld, m, w, row_base, col_base, ipiv, link);
            if (m <= 4 * kPNt)
                return launch_panel32<4, false>(ctx, st, 1, P, ld, m, w, row_base, col_base, ipiv, link);
            if (m <= 8 * 2 * kPNt)
                return launch_panel32<2, true>(ctx, st, (int)ceil_div(m, 2 * kPNt), P, ld, m, w, row_base, col_base,
                                               ipiv, link);
            return launch_panel32<4, true>(ctx, st, (int)ceil_div(m, 4 * kPNt), P, ld, m, w, row_base, col_base,
                                           ipiv, link);
        }
        if (link.moves_in || link.moves_out)
            return fail(ctx, B2M_ERR_UNSUPPORTED, "a linked FP64 panel has at most %d rows", kPMaxC * kPNt * 4);
        if (w > 16) return fail(ctx, B2M_ERR_UNSUPPORTED, "FP64 panel of %d rows needs width <= 16", m);
        if (m > panel_max_rows(true, 16)) {  // very tall: 8 columns, 8 rows per thread
            const int C = (int)ceil_div(m, kPT * 8);
            if (w > 8 || C > kPMaxC)
                return fail(ctx, B2M_ERR_UNSUPPORTED, "FP64 panel of %d x %d is too tall", m, w);
            return launch_push<T, 8, 8>(ctx, st, C, (int)ceil_div(m, C), P, ld, m, w, row_base, col_base, ipiv);
        }
        const int C = (int)ceil_div(m, kPT * 4);
        if (C > kPMaxC) return fail(ctx, B2M_ERR_UNSUPPORTED, "FP64 panel of %d rows is too tall", m);
        return launch_push<T, 16, 4>(ctx, st, C, (int)ceil_div(m, C), P, ld, m, w, row_base, col_base, ipiv);
    } else {
        static_assert(sizeof(T) == 8, "the cluster panel is instantiated for FP64 only");
        return B2M_ERR_UNSUPPORTED;
    }
}

template int32_t launch_panel<double>(Ctx*, cudaStream_t, double*, int64_t, int, int, int, int, int32_t*,
                                      const PanelLink&);

}  // namespace b2m
