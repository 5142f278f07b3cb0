// panel.cuh -- what the partial-pivoting panels share (panel.cu, zlu.cu, batched.cu).
#pragma once

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
