// The barrier of the kernels that keep a whole step of a small graph in one launch
// (phase_small.cuh, rebuild_small.cuh), and how they are launched.
#pragma once

#include "vg_internal.cuh"

constexpr int GS_THREADS = 512;
constexpr int GS_WARPS = GS_THREADS / 32;
constexpr int GS_MAX_CLUSTER = 16;

// what such a kernel leaves in pinned memory (set to GS_DONE before the launch)
enum : int32_t {
    GS_DONE = 0,
    GS_REFUSED = 1, // not a graph the kernel takes
    GS_TIMEOUT = 2, // a barrier's bounded wait ran out
    GS_ENDLESS = 3  // a phase took more iterations than a launch may (vg_ctx_set_phase_iterations)
};
// All but GS_DONE leave the graph as it was, and the general path takes it.

// All blocks of the launch reach the barrier, and what they wrote before it is visible
// after it. GRID: a counter in global memory that starts at 0 (the launch is cooperative,
// so every block is resident); a wait of `polls` reads (vg_ctx_set_barrier_polls) gives up and
// returns false in every thread of the block. A block that gave up arrives at no later barrier, so
// every other one passes the barriers it had reached, gives up at its next one and returns too.
// Else the grid is one cluster: its hardware barrier.
template <bool GRID>
__device__ __forceinline__ bool all_blocks(unsigned *arrived, unsigned &round, int &s_dead, int polls) {
    if constexpr (GRID) {
        round++;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(arrived, 1u);
            const unsigned want = round * gridDim.x;
            int read = 0;
            unsigned seen;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n"
                             : "=r"(seen)
                             : "l"(arrived)
                             : "memory");
            } while (seen < want && ++read < polls);
            if (seen < want) s_dead = 1;
            __threadfence();
        }
        __syncthreads();
        return !s_dead;
    } else {
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
        return true;
    }
}

// exclusive prefix over the warp's lanes and the warp's total
__device__ __forceinline__ int64_t warp_excl(int64_t x, int64_t &total) {
    const int lane = threadIdx.x & 31;
    int64_t s = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    total = __shfl_sync(0xffffffffu, s, 31);
    return s - x;
}

// exclusive prefix over the block's threads and the block's total
__device__ __forceinline__ int64_t block_excl(int64_t x, int64_t &total, int64_t *s_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t wt;
    const int64_t e = warp_excl(x, wt);
    if (lane == 31) s_w[warp] = wt;
    __syncthreads();
    int64_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < GS_WARPS; w++) {
        const int64_t y = s_w[w];
        before += w < warp ? y : 0;
        all += y;
    }
    __syncthreads();
    total = all;
    return before + e;
}

// The blocks a kernel pair may be launched with: the largest cluster the device takes for
// `in_cluster` and the blocks of a cooperative launch of `in_grid` (0: none). Sets the
// kernels' attributes for the current device.
template <class Args>
void vg_grid_limits(vg_ctx *ctx, void (*in_cluster)(Args), void (*in_grid)(Args), size_t smem,
                    GridLimits &lim) {
    if (lim.cluster >= 0) return;
    for (auto *k : {in_cluster, in_grid})
        VG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    VG_CUDA(cudaFuncSetAttribute(in_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    int best = 0;
    for (int size = GS_MAX_CLUSTER; size >= 1 && !best; size /= 2) {
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = size;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(size);
        cfg.blockDim = dim3(GS_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, in_cluster, &cfg) == cudaSuccess && n > 0)
            best = size;
        else
            cudaGetLastError();
    }
    int coop = 0, per_sm = 0;
    VG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
    VG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, in_grid, GS_THREADS, smem));
    lim.grid = coop && per_sm > 0 ? ctx->sm_count : 0;
    lim.cluster = best;
}

// launch over the whole device (cooperative; *arrived zeroed on the stream first) or as
// one cluster of `blocks`
template <class Args>
void vg_grid_launch(vg_ctx *ctx, void (*kernel)(Args), const Args &args, bool grid, int blocks,
                    size_t smem, unsigned *arrived) {
    if (grid) VG_CUDA(cudaMemsetAsync(arrived, 0, sizeof(unsigned), ctx->stream));
    cudaLaunchAttribute la{};
    if (grid) {
        la.id = cudaLaunchAttributeCooperative;
        la.val.cooperative = 1;
    } else {
        la.id = cudaLaunchAttributeClusterDimension;
        la.val.clusterDim.x = blocks;
        la.val.clusterDim.y = la.val.clusterDim.z = 1;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(GS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cfg.attrs = &la;
    cfg.numAttrs = 1;
    LaunchTimer lt(ctx);
    VG_CUDA(cudaLaunchKernelEx(&cfg, kernel, args));
}
