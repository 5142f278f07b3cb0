// panel.cuh -- what the partial-pivoting panels share (panel.cu, zlu.cu, batched.cu).
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace b2m {

constexpr unsigned kInfHi = 0x7ff00000u;  // leading word of infinity

// leading word of |x|
__device__ __forceinline__ uint32_t mag_hi(double x) { return (uint32_t)__double2hiint(x) & 0x7fffffffu; }

// lane of the largest a >= 0 (the lowest pos among equals), compared exactly
static __device__ __noinline__ int warp_winner(double a, int pos) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(a);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t mhi = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const bool top = hi == mhi && lo == mlo;
    const uint32_t mp = __reduce_min_sync(0xffffffffu, top ? (uint32_t)pos : 0xffffffffu);
    return __ffs(__ballot_sync(0xffffffffu, top && (uint32_t)pos == mp)) - 1;
}

// ---- Bounded waits inside a cluster.  A thread whose wait runs out notes it in every CTA's `late` word; its warp
// stops working and goes on to its CTA's next common barrier (bar_any, __syncthreads_or), where the whole CTA learns
// of it and leaves the elimination together: which barriers a thread meets never depends on what it saw alone.
// A warp that has not given up has seen every candidate so far, so what it records is always a valid interchange.

// (out of line: inlined into panel_kernel's column loop it cost 1 to 2 % of a leaf)
static __device__ __noinline__ void cluster_give_up(int* late, int C, int32_t* status, int site) {
    atomicExch(&status[kTimeout], site);
    for (int d = 0; d < C; ++d)
        asm volatile("st.shared::cluster.u32 [%0], 1;\n" ::"r"(map_rank(late, d)) : "memory");
}
// waits for a phase of this CTA's barrier, for `polls` polls or until a thread of the cluster has given up; false: in vain
__device__ __forceinline__ bool cluster_wait(uint64_t* bar, uint32_t phase, uint32_t polls, int* late, int C,
                                             int32_t* status, int site) {
    for (uint32_t it = 0; it < polls; ++it) {
        if (mbar_try_wait_cluster(bar, phase)) return true;
        if ((it & 255u) == 255u && *reinterpret_cast<volatile int*>(late) != 0) break;
    }
    cluster_give_up(late, C, status, site);
    return false;
}
// A cluster kernel's end: no CTA leaves while a push to it may be in flight.  Every push that was waited for has
// arrived.  After a wait that ran out some may not have, and nothing tells when they do, so every CTA then stays for
// about 100 us, some two hundred times what a push takes.
__device__ __forceinline__ void cluster_leave(const int* late) {
    cooperative_groups::this_cluster().sync();
    if (*reinterpret_cast<const volatile int*>(late) != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 200000) __nanosleep(200);
    }
}
// named barrier of N threads; whether any of them brought `flag`
template <int N> __device__ __forceinline__ bool bar_any(int id, bool flag) {
    uint32_t any;
    asm volatile(
        "{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.or.pred q, %2, %3, p; selp.u32 %0, 1, 0, q; }\n"
        : "=r"(any)
        : "r"(flag ? 1u : 0u), "r"(id), "n"(N)
        : "memory");
    return any != 0;
}
inline uint32_t wait_polls(const Ctx* ctx) { return ctx->wait_limit >= 0 ? (uint32_t)ctx->wait_limit : kSpinLimit; }

// One cluster of C CTAs with the critical path's priority.  plain: a kernel without cluster instructions, on one
// CTA (one with them needs the cluster attribute on a single CTA, too).
template <typename Kern, typename... Args>
int32_t launch_cluster(Ctx* ctx, cudaStream_t st, Kern kern, bool plain, int C, int threads, size_t smem, int m, int w,
                       size_t elem, Args... args) {
    // whether a cluster of C CTAs fits on this device: 1 yes, -1 no, 0 not asked yet
    std::atomic<int>& sched = device_flag((const void*)kern, 1 + C, ctx->device);
    cudaLaunchAttribute at[2];
    // the panel is the factorisation's critical path: when a look-ahead trailing update runs beside
    // it, its CTAs take free SMs ahead of the update's tiles
    at[0].id = cudaLaunchAttributePriority;
    at[0].val.priority = ctx->chain_priority;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = C;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = plain ? 1 : 2;
    if (C > 8 && sched.load() == 0) {
        int clusters = 0;
        B2M_CU(ctx, cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg));
        sched.store(clusters > 0 ? 1 : -1);
    }
    if (C > 8 && sched.load() < 0)
        return fail(ctx, B2M_ERR_UNSUPPORTED, "panel cluster of %d CTAs cannot be scheduled", C);
    prof_begin(ctx, st, kClsPanel);
    B2M_CU(ctx, cudaLaunchKernelEx(&cfg, kern, args...));
    prof_end(ctx, st, kClsPanel, 2.0 * m * w * elem);  // bytes: the panel read and written once
    B2M_LAUNCHED(ctx);
    return B2M_OK;
}

}  // namespace b2m
