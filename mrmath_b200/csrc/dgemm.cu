// dgemm.cu -- FP64 GEMM on the sm_100a DMMA path (mma.sync m16n8k4 .f64), operands staged by
// TMA into a multi-stage shared-memory ring guarded by mbarriers (one producer warp, eight
// consumer warps).  Replaces the reference's BlockMatrixMultiplication(T1/T2) + the FMA
// MatrixMultT2 inner kernel (BlockedMult.pas:350-724, FMAMatrixMultTransposedOperationsx64.pas)
// and applies the doNone/doAdd/doSub destination operation (MatrixConst.pas:147) in the epilogue.
//
// CTA tiles of 128 x 128 down to 32 x 16 (DgTile), k-step 16 doubles, 6 stages (192 KiB for the
// largest tile).  A K-major tile ([m][k], k contiguous) is loaded with the 128-byte swizzle, which
// makes the per-thread fragment loads conflict-free; an MN-major tile ([k][m or n]) is loaded
// unswizzled (one row of the tile per k).  Every element accumulates its products in ascending k,
// four at a time, whatever the tile, so the tile does not show in the result.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.cuh"

namespace b2m {
namespace {

constexpr int BKD = 16, STAGES = 6;
constexpr int kGroupM = 8;

// a CTA tile of M x N outputs on WM x WN consumer warps
template <int M, int N, int WM, int WN> struct DgTile {
    static constexpr int BM = M, BN = N, kWm = WM, kWn = WN;
    static constexpr int kTm = M / WM, kTn = N / WN;              // warp tile
    static constexpr int kI = kTm / 16, kJ = kTn / 8;             // m16n8 fragments of a warp tile
    static constexpr int kConsumerWarps = WM * WN;
    static constexpr int kThreads = (kConsumerWarps + 1) * 32;
    static constexpr int kTileA = M * BKD * 8, kTileB = N * BKD * 8, kStageBytes = kTileA + kTileB;
    static constexpr int kSmemBytes = STAGES * kStageBytes + 1024;
    static constexpr int kCtas = M >= 128 ? 1 : 2;                // CTAs per SM the registers must allow
    static_assert(kTileA % 1024 == 0 && kTileB % 1024 == 0, "swizzled tiles start on 1 KiB");
};
using DgTile128 = DgTile<128, 128, 2, 4>;
using DgTile64 = DgTile<64, 64, 2, 2>;
using DgTile32 = DgTile<32, 32, 2, 2>;
using DgTileThin = DgTile<32, 16, 2, 2>;

struct DgemmArgs {
    int M, N, K;
    int a_x0, a_y0, b_x0, b_y0;
    double* C;
    int64_t ldc;
    int op;
    int32_t* status;
    int check_info;
    int lower;  // only tiles that reach C's lower triangle (row >= column) are computed
};

__device__ __forceinline__ void dmma16x8x4(double (&d)[4], double a0, double a1, double b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ double lds64(const uint8_t* base, uint32_t off) {
    return *reinterpret_cast<const double*>(base + off);
}

template <class T, bool AK, bool BKM>
__global__ void __launch_bounds__(T::kThreads, T::kCtas)
    dgemm_tma_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, DgemmArgs p) {
    constexpr int BM = T::BM, BN = T::BN, kConsumerWarps = T::kConsumerWarps;
    constexpr int kI = T::kI, kJ = T::kJ;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES];
    __shared__ __align__(8) uint64_t empty_bar[STAGES];

    if (p.check_info && p.status[kInfo] != 0) return;  // an earlier singular pivot stops the chain

    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const int tiles_m = (p.M + BM - 1) / BM;
    const int tiles_n = (p.N + BN - 1) / BN;
    const int bid = blockIdx.x;
    const int group = bid / (kGroupM * tiles_n);
    const int first_m = group * kGroupM;
    const int gsize = min(tiles_m - first_m, kGroupM);
    const int in_group = bid % (kGroupM * tiles_n);
    const int tm = first_m + in_group % gsize;
    const int tn = in_group / gsize;

    if (p.lower && tn * BN >= (tm + 1) * BM) return;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KT = (p.K + BKD - 1) / BKD;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], kConsumerWarps);
        }
        fence_barrier_init();
    }
    __syncthreads();

    if (warp == kConsumerWarps) {
        // ---------------- producer: one elected lane issues the TMA loads
        if (lane == 0) {
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
            for (int kt = 0; kt < KT; ++kt) {
                const int s = kt % STAGES;
                const uint32_t ph = (kt / STAGES) & 1;
                if (!mbar_wait(&empty_bar[s], ph ^ 1, &p.status[kTimeout], 101)) break;
                uint8_t* sa = smem + s * T::kStageBytes;
                uint8_t* sb = sa + T::kTileA;
                mbar_arrive_expect_tx(&full_bar[s], T::kStageBytes);
                if (AK) tma_load_2d(sa, &tmA, p.a_x0 + kt * BKD, p.a_y0 + tm * BM, &full_bar[s]);
                else    tma_load_2d(sa, &tmA, p.a_x0 + tm * BM, p.a_y0 + kt * BKD, &full_bar[s]);
                if (BKM) tma_load_2d(sb, &tmB, p.b_x0 + kt * BKD, p.b_y0 + tn * BN, &full_bar[s]);
                else     tma_load_2d(sb, &tmB, p.b_x0 + tn * BN, p.b_y0 + kt * BKD, &full_bar[s]);
            }
        }
        return;
    }

    // ---------------- consumers: kWm (m) x kWn (n) warps
    const int wm = warp / T::kWn, wn = warp % T::kWn;
    const int g = lane >> 2, t = lane & 3;

    // The old destination tile is fetched into L2 while the products run (7900 x 7680, K 256: 1133 ->
    // 1070 us; the small tiles, whose operands and destination are in L2 anyway, lost 6 % to it).
    if (BM >= 128 && p.op != B2M_DO_NONE) {
        for (int e = threadIdx.x; e < BM * (BN / 16); e += kConsumerWarps * 32) {
            const int m = tm * BM + e / (BN / 16), n = tn * BN + 16 * (e % (BN / 16));
            if (m < p.M && n < p.N)
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.C + (int64_t)m * p.ldc + n));
        }
    }

    // per-thread fragment offsets (bytes within a stage tile), k4-step 0
    uint32_t offA[kI], offB[kJ];
#pragma unroll
    for (int i = 0; i < kI; ++i) {
        const int m = wm * T::kTm + i * 16 + g;
        offA[i] = AK ? (uint32_t)(m * 128 + ((t & 1) << 3)) : (uint32_t)(t * BM * 8 + m * 8);
    }
#pragma unroll
    for (int j = 0; j < kJ; ++j) {
        const int n = wn * T::kTn + j * 8 + g;
        offB[j] = BKM ? (uint32_t)(n * 128 + ((t & 1) << 3)) : (uint32_t)(t * BN * 8 + n * 8);
    }

    double acc[kI][kJ][4];
#pragma unroll
    for (int i = 0; i < kI; ++i)
#pragma unroll
        for (int j = 0; j < kJ; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

    bool ok = true;
    for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % STAGES;
        const uint32_t ph = (kt / STAGES) & 1;
        if (!mbar_wait(&full_bar[s], ph, &p.status[kTimeout], 102)) { ok = false; break; }
        const uint8_t* sa = smem + s * T::kStageBytes;
        const uint8_t* sb = sa + T::kTileA;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            double a0[kI], a1[kI], b[kJ];
#pragma unroll
            for (int i = 0; i < kI; ++i) {
                if (AK) {
                    const uint32_t o = offA[i] + ((((2 * q + (t >> 1)) ^ g) & 7) << 4);
                    a0[i] = lds64(sa, o);
                    a1[i] = lds64(sa, o + 1024);
                } else {
                    const uint32_t o = offA[i] + q * 4 * BM * 8;
                    a0[i] = lds64(sa, o);
                    a1[i] = lds64(sa, o + 64);
                }
            }
#pragma unroll
            for (int j = 0; j < kJ; ++j) {
                if (BKM) b[j] = lds64(sb, offB[j] + ((((2 * q + (t >> 1)) ^ g) & 7) << 4));
                else     b[j] = lds64(sb, offB[j] + q * 4 * BN * 8);
            }
#pragma unroll
            for (int i = 0; i < kI; ++i)
#pragma unroll
                for (int j = 0; j < kJ; ++j) dmma16x8x4(acc[i][j], a0[i], a1[i], b[j]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);
    }
    if (!ok) return;

    // ---------------- epilogue: dest op= acc, masked to the M x N operand.  The old values of a row of
    // fragments are loaded together, by pairs where the destination allows it: one at a time, each
    // behind the store before it, they cost a memory latency per element (an LU's K = 256 update of
    // 7900 x 7680 took 1479 us, 1058 without the old values; now 1070)
    const int m_base = tm * BM + wm * T::kTm;
    const int n_base = tn * BN + wn * T::kTn;
    auto store = [&](auto pairs) {  // pairs: every pair of the tile lies inside C and is 16-byte aligned
        constexpr bool kPairs = decltype(pairs)::value;
#pragma unroll
        for (int i = 0; i < kI; ++i) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = m_base + i * 16 + g + h * 8;
                if (m >= p.M) continue;
                double* c = p.C + (int64_t)m * p.ldc + n_base + 2 * t;
                const int left = p.N - n_base - 2 * t;  // columns from this thread's first one on
                double2 old[kJ];
                if (p.op != B2M_DO_NONE) {
#pragma unroll
                    for (int j = 0; j < kJ; ++j) {
                        if constexpr (kPairs) {
                            old[j] = *reinterpret_cast<const double2*>(c + 8 * j);
                        } else {
                            old[j].x = 8 * j < left ? c[8 * j] : 0.0;
                            old[j].y = 8 * j + 1 < left ? c[8 * j + 1] : 0.0;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < kJ; ++j) {
                    double2 v = make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
                    if (p.op == B2M_DO_ADD) v = make_double2(old[j].x + v.x, old[j].y + v.y);
                    if (p.op == B2M_DO_SUB) v = make_double2(old[j].x - v.x, old[j].y - v.y);
                    if constexpr (kPairs) {
                        *reinterpret_cast<double2*>(c + 8 * j) = v;
                    } else {
                        if (8 * j < left) c[8 * j] = v.x;
                        if (8 * j + 1 < left) c[8 * j + 1] = v.y;
                    }
                }
            }
        }
    };
    if ((p.ldc & 1) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0 && (tn + 1) * BN <= p.N)
        store(std::true_type{});
    else
        store(std::false_type{});
}

template <class T, bool AK, bool BKM>
int32_t launch_variant(Ctx* ctx, cudaStream_t st, const CUtensorMap& ta, const CUtensorMap& tb, const DgemmArgs& a) {
    auto kern = dgemm_tma_kernel<T, AK, BKM>;
    std::atomic<int>& attr_set = device_flag((const void*)kern, 0, ctx->device);
    if (!attr_set.load()) {
        B2M_CU(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes));
        attr_set.store(1);
    }
    const int tiles = (int)(ceil_div(a.M, T::BM) * ceil_div(a.N, T::BN));
    prof_begin(ctx, st, kClsGemm);
    B2M_CU(ctx, launch_k(ctx, kern, dim3(tiles), dim3(T::kThreads), T::kSmemBytes, st, ta, tb, a));
    prof_end(ctx, st, kClsGemm, 2.0 * a.M * a.N * a.K);
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

// the tensor maps of one tile shape, then its kernel
template <class T>
int32_t launch_tile(Ctx* ctx, cudaStream_t st, const DOperand& A, const DOperand& B, const DgemmArgs& a) {
    CUtensorMap ta, tb;
    if (A.kmajor)
        B2M_TRY(encode_tmap_2d(ctx, &ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A.base, A.cols, A.rows, A.ld * 8, BKD,
                               T::BM, CU_TENSOR_MAP_SWIZZLE_128B));
    else
        B2M_TRY(encode_tmap_2d(ctx, &ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A.base, A.cols, A.rows, A.ld * 8, T::BM,
                               BKD, CU_TENSOR_MAP_SWIZZLE_NONE));
    if (B.kmajor)
        B2M_TRY(encode_tmap_2d(ctx, &tb, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, B.base, B.cols, B.rows, B.ld * 8, BKD,
                               T::BN, CU_TENSOR_MAP_SWIZZLE_128B));
    else
        B2M_TRY(encode_tmap_2d(ctx, &tb, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, B.base, B.cols, B.rows, B.ld * 8, T::BN,
                               BKD, CU_TENSOR_MAP_SWIZZLE_NONE));
    if (A.kmajor && !B.kmajor) return launch_variant<T, true, false>(ctx, st, ta, tb, a);
    if (A.kmajor && B.kmajor) return launch_variant<T, true, true>(ctx, st, ta, tb, a);
    if (!A.kmajor && !B.kmajor) return launch_variant<T, false, false>(ctx, st, ta, tb, a);
    return launch_variant<T, false, true>(ctx, st, ta, tb, a);
}

// The tile with the smallest estimated time.  The estimates (us) are fits to the four shapes timed on
// a B200 (148 SMs; alone, event-timed, including the launch) over 30 sizes:
//   128 x 128, one CTA per SM:    9 + 0.139 K per wave           (35 TFLOP/s when the waves are full)
//   64 x 64, two per SM:          5 + 0.052 K alone on an SM, 0.076 K per wave of pairs   (32 TFLOP/s)
//   32 x 32, four per SM:         5 + 0.021 K, or 23.5 TFLOP/s over all tiles less 15 %
//   32 x 16:                      4 + 0.015 K, or 17.5 TFLOP/s less 15 %
// Measured with 128 x 128 only -> with this choice: 128^3 25.3 -> <= 14.9 us (the call's host time),
// 1500 x 256 x K 256 (an outer step of the LU) 43.1 -> 15.5, 512^3 78.5 -> 19.2, 1024^3 148 -> 84,
// 1024 x 1 x K 1024 (a residual) 147 -> 18.9, 2999 x 2777 x K 1501 889 -> 835 (subtracting); 128 x 128
// stays at 1536 x 1536 x K 320 (51 us, 64 x 64: 57) and from 4096^3 on (3986 us, 4250).  Near a line the
// estimate can miss: 7900 x 256 x K 256 takes 64 x 64 (estimated 43.9 to 44.6), 47.3 us against 43.1.
int pick_tile(const Ctx* ctx, int64_t M, int64_t N, int64_t K) {
    const double sms = ctx->num_sms, k = (double)K;
    auto tiles = [&](int tm, int tn) { return (double)(ceil_div(M, tm) * ceil_div(N, tn)); };
    const double t128 = tiles(128, 128), t64 = tiles(64, 64), t32 = tiles(32, 32), t16 = tiles(32, 16);
    const double c128 = 9 + 0.139 * k * std::ceil(t128 / sms);
    const double c64 = 5 + k * (t64 <= sms ? 0.052 : 0.076 * std::ceil(t64 / (2 * sms)));
    const double c32 = 5 + k * std::max(0.021, 1.0e-4 * t32 * (148 / sms));
    const double c16 = 4 + k * std::max(0.015, 6.7e-5 * t16 * (148 / sms));
    const double best = std::min(std::min(c128, c64), std::min(c32, c16));
    return best == c16 ? 16 : (best == c32 ? 32 : (best == c64 ? 64 : 128));
}

// C op= A(:, k0:k0+kt) B(k0:k0+kt, :) for a short k range (kt < 16): the tail of a K that ends inside
// the operands' tensor maps, where the 16-wide TMA k-tile would read other data.  One thread per
// output, K FMAs each; these tails are narrow (the 8-column leaves of very tall factorisations).
__global__ void dgemm_ktail_kernel(const double* A, int64_t lda, int64_t ar0, int64_t ac0, int akmajor,
                                   const double* B, int64_t ldb, int64_t br0, int64_t bc0, int bkmajor, double* C,
                                   int64_t ldc, int M, int N, int k0, int kt, int op, const int32_t* status,
                                   int check_info) {
    if (check_info && status[kInfo] != 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)M * N) return;
    const int m = (int)(e / N), n = (int)(e - (int64_t)m * N);
    double s = 0.0;
    for (int k = k0; k < k0 + kt; ++k) {
        const double a = akmajor ? A[(ar0 + m) * lda + ac0 + k] : A[(ar0 + k) * lda + ac0 + m];
        const double b = bkmajor ? B[(br0 + n) * ldb + bc0 + k] : B[(br0 + k) * ldb + bc0 + n];
        s = fma(a, b, s);
    }
    double* c = C + (int64_t)m * ldc + n;
    *c = op == B2M_DO_NONE ? s : (op == B2M_DO_ADD ? *c + s : *c - s);
}

}  // namespace

int32_t dgemm_tiled(Ctx* ctx, cudaStream_t st, const DOperand& A, const DOperand& B, double* C, int64_t ldc, int64_t M,
                    int64_t N, int64_t K, int op, bool check_info, bool lower) {
    if (M <= 0 || N <= 0) return B2M_OK;
    if (K <= 0) {
        if (op == B2M_DO_NONE) B2M_CU(ctx, cudaMemset2DAsync(C, ldc * 8, 0, N * 8, M, st));
        return B2M_OK;
    }
    // A K that is not a multiple of the 16-wide k-tile is safe only where the k range ends at the
    // tensor maps' extent (TMA fills beyond it with zeros); elsewhere the last partial k-tile runs
    // as a separate short-K pass after the tiled product of the first K - K % 16.
    const int64_t a_kend = A.kmajor ? A.c0 + K : A.r0 + K, a_ext = A.kmajor ? A.cols : A.rows;
    const int64_t b_kend = B.kmajor ? B.c0 + K : B.r0 + K, b_ext = B.kmajor ? B.cols : B.rows;
    if ((K & 15) && (a_kend != a_ext || b_kend != b_ext)) {
        const int64_t K16 = K & ~int64_t(15);
        int tail_op = op;
        if (K16 > 0) {
            B2M_TRY(dgemm_tiled(ctx, st, A, B, C, ldc, M, N, K16, op, check_info, lower));
            if (op == B2M_DO_NONE) tail_op = B2M_DO_ADD;
        }
        const int64_t outs = M * N;
        prof_begin(ctx, st, kClsGemm);
        B2M_CU(ctx, launch_k(ctx, dgemm_ktail_kernel, dim3((unsigned)ceil_div(outs, 256)), dim3(256), 0, st,
                             static_cast<const double*>(A.base), A.ld, A.r0, A.c0, A.kmajor ? 1 : 0,
                             static_cast<const double*>(B.base), B.ld, B.r0, B.c0, B.kmajor ? 1 : 0, C, ldc, (int)M,
                             (int)N, (int)K16, (int)(K - K16), tail_op, ctx->d_status, check_info ? 1 : 0));
        prof_end(ctx, st, kClsGemm, 2.0 * M * N * (K - K16));
        B2M_LAUNCHED(ctx);
        return B2M_OK;
    }
    if ((A.c0 & 1) || (B.c0 & 1) || (A.ld & 1) || (B.ld & 1))
        return fail(ctx, B2M_ERR_DIM, "dgemm_tiled: TMA origin/stride must be even (A.c0=%lld B.c0=%lld)",
                    (long long)A.c0, (long long)B.c0);
    DgemmArgs a;
    a.M = (int)M; a.N = (int)N; a.K = (int)K;
    a.a_x0 = (int)A.c0; a.a_y0 = (int)A.r0;
    a.b_x0 = (int)B.c0; a.b_y0 = (int)B.r0;
    a.C = C; a.ldc = ldc; a.op = op;
    a.status = ctx->d_status;
    a.check_info = check_info ? 1 : 0;
    a.lower = lower ? 1 : 0;
    switch (pick_tile(ctx, M, N, K)) {
        case 128: return launch_tile<DgTile128>(ctx, st, A, B, a);
        case 64: return launch_tile<DgTile64>(ctx, st, A, B, a);
        case 32: return launch_tile<DgTile32>(ctx, st, A, B, a);
        default: return launch_tile<DgTileThin>(ctx, st, A, B, a);
    }
}

}  // namespace b2m
