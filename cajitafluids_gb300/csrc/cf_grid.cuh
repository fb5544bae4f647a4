// Grid-wide barriers and folds of the on-chip solves (cf_pcg.cu, cf_cg32.cu):
// one cooperative launch runs many solver iterations, its blocks meeting at
// barriers in global memory.
#pragma once
#include "cf_ctx.cuh"

namespace cf {

// polls of a grid barrier before the launch gives up (each poll is an L2
// round trip; a barrier takes a few of them)
constexpr unsigned PC_WAIT_LIMIT = 1u << 22;
constexpr unsigned PC_STALL_LIMIT = 1u << 10;

// Grid barrier in two halves (all blocks co-resident: cooperative launch).
// The counter only grows: S->gbar is its value when the launch starts.
__device__ __forceinline__ void grid_arrive(SolverState* S) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&S->gcount) : "memory");
    }
}
// true when the arrivals have reached target; the wait is bounded, and ends
// early once another block has given up.  stall: the timeout-path test's wait
// (cf_test_stall_wait), for arrivals that never come.
__device__ __forceinline__ bool grid_wait(SolverState* S, unsigned target, bool stall = false) {
    bool ok = true;
    if (threadIdx.x == 0) {
        const unsigned limit = stall ? PC_STALL_LIMIT : PC_WAIT_LIMIT;
        if (stall) target += 1u << 30;
        unsigned v, k = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&S->gcount) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((k & 255u) == 255u && *(volatile int*)&S->status == ST_TIMEOUT) break;
        } while (++k < limit);
        ok = (int)(v - target) >= 0;
        if (!ok) atomicExch(&S->status, (int)ST_TIMEOUT);
    }
    return __syncthreads_and(ok);
}

// The strided part of final_trees over n unit partials: thread t of the 256
// adds partial[t], partial[t + 256], ... in that order.
__device__ __forceinline__ double strided_sum(const double* part, int n, int t) {
    double s = 0.0;
    for (int u = t; u < n; u += CF_RED_THREADS) s = s + __ldcg(part + u);
    return s;
}

// a cooperative launch (every block resident)
template <typename... P, typename... A>
inline cudaError_t launch_all(void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t stream,
                              const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
// whether that many blocks are resident at once (and the shared memory granted)
template <typename... P>
inline bool all_fit(void (*kernel)(P...), int blocks, int threads, size_t smem, int sms) {
    int occ = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return occ * sms >= blocks;
}

}  // namespace cf
