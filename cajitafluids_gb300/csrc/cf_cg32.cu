// FP32 inner Jacobi-PCG iteration of the mixed-precision projection, fed by
// TMA.
//
// The FP32 solver vectors (r, p twice) carry a one-cell ghost ring:
// element (i, j), i in [-1, nx], j in [-1, ny], lives at
// base[(j + 1) * pitch + i + 4], so owned column 0 sits on a 16-byte boundary.
// Wall ghosts stay zero; along a periodic axis the thread that writes an
// edge cell also writes its ghost copy, so every halo a kernel reads was
// written by an earlier launch.
//
// Each kernel is persistent (two CTAs per SM).  A CTA walks tiles of 128 x 16
// owned cells; for each tile a single thread issues 2-D TMA copies
// (cp.async.bulk.tensor) of 136 x 18 boxes -- the tile, one halo row above and
// below and a 4-column (16-byte) pad on each side -- into one of three
// shared-memory stages, completing on an mbarrier.  While a tile is computed
// from shared memory the next two are in flight.  Stores go straight from
// registers (float4 where a full vector is owned).
//
//   K1  p <- M^-1 r + beta p (halo too, in shared memory) ; q <- A p ; p.q
//   K2  q <- A p (recomputed) ; x += alpha p (double-float) ; r -= alpha q ;
//       r.z , r.r
//
// Dot products: FP32 per thread within a tile, FP64 across tiles, warps and
// CTAs; the last CTA finishes the sum and advances the solver state.
// mbarrier waits are bounded: on timeout the CTA records ST_TIMEOUT, waits
// (bounded) for its own copies still in flight, and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "cf_grid.cuh"

namespace cf {

#define FULLMASK32 0xffffffffu

constexpr int kTW = 128;                 // owned columns per tile
constexpr int kTH = 16;                  // owned rows per tile
constexpr int kBX = kTW + 8;             // box columns
constexpr int kBY = kTH + 2;             // box rows
constexpr int kBoxBytes = kBX * kBY * 4; // 9792
constexpr int kSlot = 9856;              // 128-byte aligned slot
constexpr int kStages = 3;
constexpr int kThreads = 256;
// CTAs to an SM of K1 and K2: the FP32 sums of a CTA's tiles follow the grid, so it is
// fixed here rather than left to the registers a build happens to need
constexpr int kCtas1 = 3, kCtas2 = 2;
constexpr unsigned kWaitLimit = 1u << 22;
// the drain after a timeout waits longer than any tile wait: a CTA must not
// exit while one of its bulk copies may still be writing its shared memory
constexpr unsigned kDrainLimit = 1u << 24;
// the stalled wait of the timeout-path test (cf_test_stall_wait)
constexpr unsigned kStallLimit = 1u << 10;

struct Cg32T {
    int nx, ny, per_x, per_y, tiles_x, tiles, pitch;
    int mg;  // MG-PCG: K1 reads z (minv = 1), K2 leaves beta and rho to k_mg_rz32
    Stencil st;
    float *r, *pa, *pb;  // element (0, 0)
    float2* x;           // the solution as double-float pairs (owned cells, row pitch xpitch)
    int xpitch;
    double *part0, *part1;
    SolverState* S;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait; true when the phase completed
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned limit) {
    for (unsigned k = 0; k < limit; ++k)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ int ebits32t(const Cg32T& a, int i, int j) {
    int ci = wrap_index(i, a.nx, a.per_x), cj = wrap_index(j, a.ny, a.per_y);
    if (ci < 0) ci = 0;
    if (cj < 0) cj = 0;
    return edge_bits(ci, cj, a.nx, a.ny, a.per_x, a.per_y);
}

// store one owned value and, along a periodic axis, its ghost copy
__device__ __forceinline__ void put_ghosted(const Cg32T& a, float* o, int i, int j, float val) {
    const ptrdiff_t row = (ptrdiff_t)j * a.pitch;
    o[row + i] = val;
    if (a.per_x) {
        if (i == 0) o[row + a.nx] = val;
        if (i == a.nx - 1) o[row - 1] = val;
    }
    if (a.per_y) {
        if (j == 0) o[(ptrdiff_t)a.ny * a.pitch + i] = val;
        if (j == a.ny - 1) o[-(ptrdiff_t)a.pitch + i] = val;
    }
}

// store four consecutive owned values starting at column i
__device__ __forceinline__ void put4(const Cg32T& a, float* o, int i, int j, float4 v, bool ghosts) {
    if (i + 3 < a.nx) {
        *reinterpret_cast<float4*>(o + (ptrdiff_t)j * a.pitch + i) = v;
        if (ghosts && ((a.per_x && (i == 0 || i + 3 == a.nx - 1)) || (a.per_y && (j == 0 || j == a.ny - 1)))) {
            put_ghosted(a, o, i, j, v.x);
            put_ghosted(a, o, i + 1, j, v.y);
            put_ghosted(a, o, i + 2, j, v.z);
            put_ghosted(a, o, i + 3, j, v.w);
        }
        return;
    }
    float vv[4] = {v.x, v.y, v.z, v.w};
    for (int k = 0; k < 4; ++k)
        if (i + k < a.nx) {
            if (ghosts)
                put_ghosted(a, o, i + k, j, vv[k]);
            else
                o[(ptrdiff_t)j * a.pitch + i + k] = vv[k];
        }
}

__device__ __forceinline__ float stencil1(const Cg32T& a, int i, int j, float c, float w, float e, float s, float n) {
    float q = a.st.diag32[ebits32t(a, i, j)] * c;
    q = fmaf(a.st.ms32, w, q);
    q = fmaf(a.st.ms32, e, q);
    q = fmaf(a.st.ms32, s, q);
    q = fmaf(a.st.ms32, n, q);
    return q;
}

// A p for the four cells (i0..i0+3, j) of a lane from the shared tile P
// (row stride kBX, owned (c, r) at [r + 1][c + 4]).
template <bool INTERIOR>
__device__ __forceinline__ float4 apply4(const Cg32T& a, const float* P, int lane, int row, int i0, int j,
                                         float4& pc) {
    const float* rc = P + (row + 1) * kBX + 4 + 4 * lane;
    pc = *reinterpret_cast<const float4*>(rc);
    float4 pu = *reinterpret_cast<const float4*>(rc - kBX);
    float4 pd = *reinterpret_cast<const float4*>(rc + kBX);
    float left = __shfl_up_sync(FULLMASK32, pc.w, 1);
    float right = __shfl_down_sync(FULLMASK32, pc.x, 1);
    if (lane == 0) left = rc[-1];
    if (lane == 31) right = rc[4];
    float4 q;
    if (INTERIOR) {
        const float d0 = a.st.diag32[0], ms = a.st.ms32;
        q.x = fmaf(ms, pd.x, fmaf(ms, pu.x, fmaf(ms, pc.y, fmaf(ms, left, d0 * pc.x))));
        q.y = fmaf(ms, pd.y, fmaf(ms, pu.y, fmaf(ms, pc.z, fmaf(ms, pc.x, d0 * pc.y))));
        q.z = fmaf(ms, pd.z, fmaf(ms, pu.z, fmaf(ms, pc.w, fmaf(ms, pc.y, d0 * pc.z))));
        q.w = fmaf(ms, pd.w, fmaf(ms, pu.w, fmaf(ms, right, fmaf(ms, pc.z, d0 * pc.w))));
    } else {
        q.x = stencil1(a, i0, j, pc.x, left, pc.y, pu.x, pd.x);
        q.y = stencil1(a, i0 + 1, j, pc.y, pc.x, pc.z, pu.y, pd.y);
        q.z = stencil1(a, i0 + 2, j, pc.z, pc.y, pc.w, pu.z, pd.z);
        q.w = stencil1(a, i0 + 3, j, pc.w, pc.z, right, pu.w, pd.w);
    }
    return q;
}

// true when no cell of the tile or of its halo is next to a wall: every
// diagonal and preconditioner entry is then the interior value
__device__ __forceinline__ bool interior_tile(const Cg32T& a, int i0, int j0) {
    bool wx = !a.per_x && (i0 <= 1 || i0 + kTW >= a.nx - 1);
    bool wy = !a.per_y && (j0 <= 1 || j0 + kTH >= a.ny - 1);
    bool full = i0 + kTW <= a.nx && j0 + kTH <= a.ny;
    return full && !(wx || wy);
}

__device__ __forceinline__ bool running(const SolverState* S) {
    return *(volatile const int*)&S->status == ST_RUNNING && *(volatile const int*)&S->inner_status == ST_RUNNING;
}

__device__ __forceinline__ double block_sum(double v, double* red) {
    v = warp_fold(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = red[0];
    for (int k = 1; k < kThreads / 32; ++k) t = t + red[k];
    __syncthreads();
    return t;
}

// Timeout path: record the status and wait (bounded, with the longer drain
// limit) for this CTA's copies still in flight.
__device__ void abandon(SolverState* S, const uint64_t* bars, int kfirst, int ktiles) {
    if (threadIdx.x == 0) {
        atomicExch(&S->status, (int)ST_TIMEOUT);
        for (int k = kfirst; k < ktiles && k < kfirst + kStages; ++k)
            mbar_wait(smem_u32(&bars[k % kStages]), (uint32_t)((k / kStages) & 1), kDrainLimit);
    }
    __syncthreads();
}

// K1: new direction (with halo) in shared memory, stencil, p.q.  MG: on z, whose
// preconditioner is the identity.
template <bool MG>
__global__ void __launch_bounds__(kThreads, MG ? 4 : kCtas1)
    k_tma_dir_matvec32(const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_pa,
                       const __grid_constant__ CUtensorMap map_pb, Cg32T a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[kStages];
    // test knob: an mbarrier that nothing arrives on (cf_test_stall_wait)
    __shared__ __align__(8) uint64_t never;
    __shared__ double red[kThreads / 32];
    __shared__ SolverState Z;  // the state on entry
    SolverState* S = a.S;
    copy_state(&Z, S);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(smem_u32(&bars[s]), 1);
        mbar_init(smem_u32(&never), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (Z.status != ST_RUNNING || Z.inner_status != ST_RUNNING) return;
    const int it = Z.inner_iter;
    const bool first = it == 0 || Z.restart;
    const bool stall = Z.test_stall != 0 && blockIdx.x == 0;
    const float beta = (float)Z.beta_in;
    const CUtensorMap* map_old = (it & 1) ? &map_pb : &map_pa;
    float* pnew = (it & 1) ? a.pa : a.pb;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntile = (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    unsigned char* sb = smem + ((128u - (smem_u32(smem) & 127u)) & 127u);  // TMA wants 128-byte slots
    auto stage_ptr = [&](int s, int arr) { return reinterpret_cast<float*>(sb + (s * 2 + arr) * kSlot); };
    auto issue = [&](int k) {
        int t = (int)blockIdx.x + k * (int)gridDim.x;
        int s = k % kStages;
        int x = (t % a.tiles_x) * kTW, y = (t / a.tiles_x) * kTH;
        uint32_t bar = smem_u32(&bars[s]);
        mbar_expect_tx(bar, 2 * kBoxBytes);
        tma_load_2d(smem_u32(stage_ptr(s, 0)), &map_r, x, y, bar);
        tma_load_2d(smem_u32(stage_ptr(s, 1)), map_old, x, y, bar);
    };
    if (tid == 0)
        for (int k = 0; k < kStages && k < ntile; ++k) issue(k);
    float acc = 0.f;  // FP32 over this block's tiles (no FP64 in the loop)
    for (int k = 0; k < ntile; ++k) {
        const int s = k % kStages;
        const int t = (int)blockIdx.x + k * (int)gridDim.x;
        const int i0 = (t % a.tiles_x) * kTW, j0 = (t / a.tiles_x) * kTH;
        // with the test knob, block 0's first wait is on the barrier nothing
        // arrives on, with a short limit: it times out, and the drain below
        // waits for the real copies of stages 0..2
        bool ok = (stall && k == 0) ? mbar_wait(smem_u32(&never), 0u, kStallLimit)
                                    : mbar_wait(smem_u32(&bars[s]), (uint32_t)((k / kStages) & 1), kWaitLimit);
        if (__syncthreads_or(!ok)) {
            abandon(S, bars, k, ntile);
            return;
        }
        float* R = stage_ptr(s, 0);
        float* P = stage_ptr(s, 1);
        const bool inner = interior_tile(a, i0, j0);
        // phase 1: P <- M^-1 R + beta P over the whole box (halo included)
        for (int v = tid; v < kBY * (kBX / 4); v += kThreads) {
            float4 rv = reinterpret_cast<float4*>(R)[v];
            float4 pv = reinterpret_cast<float4*>(P)[v];
            float4 o;
            if (MG) {
                o = rv;
            } else if (inner) {
                const float m0 = a.st.minv32[0];
                o.x = m0 * rv.x;
                o.y = m0 * rv.y;
                o.z = m0 * rv.z;
                o.w = m0 * rv.w;
            } else {
                int row = v / (kBX / 4), c4 = v % (kBX / 4);
                int j = j0 - 1 + row, i = i0 - 4 + 4 * c4;
                o.x = a.st.minv32[ebits32t(a, i, j)] * rv.x;
                o.y = a.st.minv32[ebits32t(a, i + 1, j)] * rv.y;
                o.z = a.st.minv32[ebits32t(a, i + 2, j)] * rv.z;
                o.w = a.st.minv32[ebits32t(a, i + 3, j)] * rv.w;
            }
            if (!first) {
                o.x = fmaf(beta, pv.x, o.x);
                o.y = fmaf(beta, pv.y, o.y);
                o.z = fmaf(beta, pv.z, o.z);
                o.w = fmaf(beta, pv.w, o.w);
            }
            reinterpret_cast<float4*>(P)[v] = o;
        }
        __syncthreads();
        // phase 2: q = A p on the owned cells, p.q, store p
        float part = 0.f;
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int row = 2 * warp + rr, j = j0 + row, i = i0 + 4 * lane;
            float4 pc;
            float4 q = inner ? apply4<true>(a, P, lane, row, i, j, pc) : apply4<false>(a, P, lane, row, i, j, pc);
            if (j < a.ny && i < a.nx) {
                part = fmaf(pc.x, q.x, part);
                if (i + 1 < a.nx) part = fmaf(pc.y, q.y, part);
                if (i + 2 < a.nx) part = fmaf(pc.z, q.z, part);
                if (i + 3 < a.nx) part = fmaf(pc.w, q.w, part);
                put4(a, pnew, i, j, pc, true);
            }
        }
        acc = acc + part;
        fence_proxy_async();
        __syncthreads();
        if (tid == 0 && k + kStages < ntile) issue(k + kStages);
    }
    double pq;
    bool finish;
    if (MG) {
        double v[1] = {warp_fold((double)acc)};
        finish = grid_totals<1, kThreads / 32>(v, a.part0, nullptr, &S->ticket[5]);
        pq = v[0];
    } else {
        const double tot = block_sum((double)acc, red);
        if (tid == 0) a.part0[blockIdx.x] = tot;
        finish = last_block_arrive(&S->ticket[5]);
        if (finish) pq = final_tree(a.part0, gridDim.x);
    }
    if (finish) {
        if (tid == 0) {
            S->ticket[5] = 0;
            S->restart = 0;
            if (isnan(pq))
                S->status = ST_NAN;
            else if (!(pq > 0.0))
                S->inner_status = ST_BREAKDOWN;  // FP32 noise floor: refine and restart
            else
                S->alpha_in = Z.rho_in / pq;
        }
    }
}

// K2: recompute A p, update x (double-float) and r, r.z and r.r.  x is read
// with plain loads issued before the tile's copies are awaited.
__global__ void __launch_bounds__(kThreads, kCtas2)
    k_tma_update32(const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_pa,
                   const __grid_constant__ CUtensorMap map_pb, Cg32T a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[kStages];
    __shared__ double red[kThreads / 32];
    SolverState* S = a.S;
    if (!running(S)) return;
    const int it = S->inner_iter;
    const CUtensorMap* map_p = (it & 1) ? &map_pa : &map_pb;
    const float alpha = (float)S->alpha_in, malpha = -alpha;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntile = (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    unsigned char* sb = smem + ((128u - (smem_u32(smem) & 127u)) & 127u);  // TMA wants 128-byte slots
    auto stage_ptr = [&](int s, int arr) { return reinterpret_cast<float*>(sb + (s * 2 + arr) * kSlot); };
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(smem_u32(&bars[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue = [&](int k) {
        int t = (int)blockIdx.x + k * (int)gridDim.x;
        int s = k % kStages;
        int x = (t % a.tiles_x) * kTW, y = (t / a.tiles_x) * kTH;
        uint32_t bar = smem_u32(&bars[s]);
        mbar_expect_tx(bar, 2 * kBoxBytes);
        tma_load_2d(smem_u32(stage_ptr(s, 0)), map_p, x, y, bar);
        tma_load_2d(smem_u32(stage_ptr(s, 1)), &map_r, x, y, bar);
    };
    if (tid == 0)
        for (int k = 0; k < kStages && k < ntile; ++k) issue(k);
    float arz = 0.f, arr = 0.f;  // FP32 over this block's tiles (no FP64 in the loop)
    for (int k = 0; k < ntile; ++k) {
        const int s = k % kStages;
        const int t = (int)blockIdx.x + k * (int)gridDim.x;
        const int i0 = (t % a.tiles_x) * kTW, j0 = (t / a.tiles_x) * kTH;
        const bool inner = interior_tile(a, i0, j0);
        // x of the lane's cells (i .. i + 3) on its two rows
        float4 xv[2][2];
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int j = j0 + 2 * warp + rr, i = i0 + 4 * lane;
            const float2* xp = a.x + (size_t)j * a.xpitch + i;
            if (inner) {
                xv[rr][0] = reinterpret_cast<const float4*>(xp)[0];
                xv[rr][1] = reinterpret_cast<const float4*>(xp)[1];
            } else {
                float* xf = reinterpret_cast<float*>(xv[rr]);
                for (int c = 0; c < 4; ++c) {
                    const bool in = j < a.ny && i + c < a.nx;
                    const float2 v = in ? xp[c] : make_float2(0.f, 0.f);
                    xf[2 * c] = v.x;
                    xf[2 * c + 1] = v.y;
                }
            }
        }
        bool ok = mbar_wait(smem_u32(&bars[s]), (uint32_t)((k / kStages) & 1), kWaitLimit);
        if (__syncthreads_or(!ok)) {
            abandon(S, bars, k, ntile);
            return;
        }
        const float* P = stage_ptr(s, 0);
        const float* R = stage_ptr(s, 1);
        float prz = 0.f, prr = 0.f;
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int row = 2 * warp + rr, j = j0 + row, i = i0 + 4 * lane;
            float4 pc;
            float4 q = inner ? apply4<true>(a, P, lane, row, i, j, pc) : apply4<false>(a, P, lane, row, i, j, pc);
            const int off = (row + 1) * kBX + 4 + 4 * lane;
            float4 rv = *reinterpret_cast<const float4*>(R + off);
            float2 x0 = df_add_f(make_float2(xv[rr][0].x, xv[rr][0].y), alpha * pc.x);
            float2 x1 = df_add_f(make_float2(xv[rr][0].z, xv[rr][0].w), alpha * pc.y);
            float2 x2 = df_add_f(make_float2(xv[rr][1].x, xv[rr][1].y), alpha * pc.z);
            float2 x3 = df_add_f(make_float2(xv[rr][1].z, xv[rr][1].w), alpha * pc.w);
            rv.x = fmaf(malpha, q.x, rv.x);
            rv.y = fmaf(malpha, q.y, rv.y);
            rv.z = fmaf(malpha, q.z, rv.z);
            rv.w = fmaf(malpha, q.w, rv.w);
            if (inner) {
                const float m0 = a.st.minv32[0];
                float s2 = fmaf(rv.w, rv.w, fmaf(rv.z, rv.z, fmaf(rv.y, rv.y, rv.x * rv.x)));
                prr += s2;
                prz = fmaf(m0, s2, prz);
                float4* xo = reinterpret_cast<float4*>(a.x + (size_t)j * a.xpitch + i);
                xo[0] = make_float4(x0.x, x0.y, x1.x, x1.y);
                xo[1] = make_float4(x2.x, x2.y, x3.x, x3.y);
                put4(a, a.r, i, j, rv, true);
            } else if (j < a.ny && i < a.nx) {
                float rvs[4] = {rv.x, rv.y, rv.z, rv.w};
                const float2 xs[4] = {x0, x1, x2, x3};
                float2* xo = a.x + (size_t)j * a.xpitch + i;
                for (int c = 0; c < 4; ++c)
                    if (i + c < a.nx) {
                        float z = a.st.minv32[ebits32t(a, i + c, j)] * rvs[c];
                        prz = fmaf(rvs[c], z, prz);
                        prr = fmaf(rvs[c], rvs[c], prr);
                        xo[c] = xs[c];
                    }
                put4(a, a.r, i, j, rv, true);
            }
        }
        arz = arz + prz;
        arr = arr + prr;
        __syncthreads();
        if (tid == 0 && k + kStages < ntile) issue(k + kStages);
    }
    double trz = block_sum((double)arz, red);
    double trr = block_sum((double)arr, red);
    if (tid == 0) {
        a.part0[blockIdx.x] = trz;
        a.part1[blockIdx.x] = trr;
    }
    if (last_block_arrive(&S->ticket[6])) {
        double sums[2];
        final_trees<2>(a.part0, a.part1, gridDim.x, sums);
        const double rz = sums[0], rr = sums[1];
        if (tid == 0) {
            S->ticket[6] = 0;
            S->rho_prev = S->rho_in;
            if (!a.mg) {
                S->beta_in = rz / S->rho_in;
                S->rho_in = rz;
            }
            S->rr_in = rr;
            if (rr > S->rr_in0) S->rr_in0 = rr;
            S->inner_iter = it + 1;
            S->iter = S->iter + 1;
            // reliable update when the recursive residual fell by delta since
            // the last one, or already looks converged
            if (isnan(rr))
                S->status = ST_NAN;
            else if (rr <= S->tau2 * S->rr_in0 || rr <= S->target2)
                S->inner_status = ST_CONVERGED;
            else if (S->iter >= S->max_iter)
                S->inner_status = ST_MAXIT;
        }
    }
}

// --------------------------------------------------------------------------
// The same iteration with the whole solve on chip, for grids of at most four
// tiles per SM (about 1.2 million cells): one cooperative launch runs many
// iterations, a block keeping its tiles' r, x and A p in registers and p with its
// halo in shared memory, the grid meeting at two barriers per iteration
// (cf_grid.cuh).  The launches above cost 22 us per iteration at 501 x 333 (84
// tiles), most of it launch, TMA and fold latency; this form 8.2 us, half of it
// the two barriers and half the FP64 sums and divisions between them.  Every cell value, thread sum,
// block sum and fold is formed as by those kernels (tile k of block b is tile
// b + k gridDim; the thread sums of tiles that one of their blocks walks in turn
// run on in the same order), so the results are the same bits.
constexpr int kHalo = 2 * kTW + 2 * kTH;  // halo (and border) values of a tile
constexpr int kMaxTiles = 4;              // tiles per block

template <int NT>
__global__ void __launch_bounds__(kThreads, 1) k_pcg32(Cg32T a, float* border, int ga, int gb, int iters) {
    extern __shared__ __align__(16) float Ps[];  // NT tiles of kBY rows of kBX columns, owned (c, r) at [r + 1][c + 4]
    __shared__ float tab_d[16], tab_m[16];
    __shared__ double red[2][NT][kThreads / 32], ws0[kThreads / 32], ws1[kThreads / 32];
    __shared__ double bc_a, bc_b, bc_c;
    __shared__ float bc_f;  // alpha, then beta, in FP32 (one conversion)
    __shared__ int bc_stat;
    SolverState* S = a.S;
    if (!running(S)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x;
    int it = S->inner_iter, iter = S->iter;
    const int it_end = it + iters, max_iter = S->max_iter;
    bool first = it == 0 || S->restart;
    double rho = S->rho_in, rho_prev = S->rho_prev, rr = S->rr_in, rr0 = S->rr_in0, alpha64 = S->alpha_in,
           beta64 = S->beta_in;
    const bool stall = S->test_stall != 0 && blockIdx.x == 0;
    const unsigned gbase = S->gbar;
    unsigned arrived = 0;
    if (tid < 16) {
        tab_d[tid] = a.st.diag32[tid];
        tab_m[tid] = a.st.minv32[tid];
    }
    for (int k = tid; k < NT * kBY * kBX; k += kThreads) Ps[k] = 0.f;
    __syncthreads();
    const float ms = a.st.ms32;
    auto tile_of = [&](int k) { return (int)blockIdx.x + k * nb; };
    auto P = [&](int k) { return Ps + k * kBY * kBX; };
    // the lane's cells: columns 4 lane .. 4 lane + 3 of rows 2 warp, 2 warp + 1
    float2 x[NT][2][4];
    float4 r[NT][2], q[NT][2];
    unsigned code[NT];    // 4 wall-adjacency bits per cell
    unsigned valid[NT];   // a bit per cell in the grid; bit 31: no wall near the tile
    int hsrc[NT][2];      // border values this thread reads (-1: none, a wall)
    short hpos[NT][2];    // and their places in the tile
    float zh[NT][2];
    const float* pold = (it & 1) ? a.pb : a.pa;
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const int t = tile_of(k), i0 = (t % a.tiles_x) * kTW, j0 = (t / a.tiles_x) * kTH;
        const bool on = t < a.tiles;
        const int nc = min(kTW, a.nx - i0), nr = min(kTH, a.ny - j0);
        code[k] = 0;
        valid[k] = on && interior_tile(a, i0, j0) ? 1u << 31 : 0u;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const int row = 2 * warp + y, j = j0 + row;
            float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int i = i0 + 4 * lane + c;
                x[k][y][c] = make_float2(0.f, 0.f);
                if (on && i < a.nx && j < a.ny) {
                    code[k] |= (unsigned)edge_bits(i, j, a.nx, a.ny, a.per_x, a.per_y) << (4 * (4 * y + c));
                    valid[k] |= 1u << (4 * y + c);
                    v[c] = a.r[(ptrdiff_t)j * a.pitch + i];
                    x[k][y][c] = a.x[(size_t)j * a.xpitch + i];
                    if (!first) P(k)[(row + 1) * kBX + 4 + 4 * lane + c] = pold[(ptrdiff_t)j * a.pitch + i];
                }
            }
            r[k][y] = make_float4(v[0], v[1], v[2], v[3]);
            q[k][y] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // halo: the row below and above, the column west and east of the tile's
        // cells in the grid; in the owner's border they are its last row, first
        // row, last column, first column
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = tid + h * kThreads;
            hsrc[k][h] = -1;
            hpos[k][h] = 0;
            zh[k][h] = 0.f;
            if (!on || e >= kHalo) continue;
            int gc, gj, pos, off;
            bool in;
            if (e < 2 * kTW) {
                const int c = e % kTW, up = e / kTW;
                in = c < nc;
                gc = i0 + c;
                gj = up ? j0 + nr : j0 - 1;
                pos = (up ? nr + 1 : 0) * kBX + 4 + c;
                off = (up ? 0 : kTW) + c;
            } else {
                const int y = (e - 2 * kTW) % kTH, east = (e - 2 * kTW) / kTH;
                in = y < nr;
                gj = j0 + y;
                gc = east ? i0 + nc : i0 - 1;
                pos = (y + 1) * kBX + 4 + (east ? nc : -1);
                off = 2 * kTW + (east ? 0 : kTH) + y;
            }
            const int wc = wrap_index(gc, a.nx, a.per_x), wj = wrap_index(gj, a.ny, a.per_y);
            if (!in || wc < 0 || wj < 0) continue;
            hsrc[k][h] = ((wj / kTH) * a.tiles_x + wc / kTW) * kHalo + off;
            hpos[k][h] = (short)pos;
            const ptrdiff_t o = (ptrdiff_t)wj * a.pitch + wc;
            zh[k][h] = tab_m[edge_bits(wc, wj, a.nx, a.ny, a.per_x, a.per_y)] * a.r[o];
            if (!first) P(k)[pos] = pold[o];
        }
    }
    __syncthreads();
    // tiles of one block of the launch-per-phase kernels (ga and gb blocks there)
    // add their thread sums up in turn
    const int na = ga < a.tiles ? ga / nb : NT, nbb = gb < a.tiles ? gb / nb : NT;
    auto add_to = [&](float (&acc)[NT], int k, int n, float v) {
#pragma unroll
        for (int g = 0; g < NT; ++g)
            if (k % n == g) acc[g] = acc[g] + v;
    };
    auto warp_sums = [&](const float (&acc)[NT], int n, double (*out)[kThreads / 32]) {
#pragma unroll
        for (int g = 0; g < NT; ++g)
            if (g < n && tile_of(g) < a.tiles) {
                const double v = warp_fold((double)acc[g]);
                if (lane == 0) out[g][warp] = v;
            }
    };
    auto put_partial = [&](const double (*w)[kThreads / 32], int g, int n, double* part) {
        if (g < n && tile_of(g) < a.tiles && lane == 0) {
            double t = w[g][0];
            for (int k = 1; k < kThreads / 32; ++k) t = t + w[g][k];
            __stcg(part + tile_of(g), t);
        }
    };
    double* const partA = a.part0;
    double* const partB0 = a.part0 + a.tiles;
    double* const partB1 = partB0 + a.tiles;
    const int nwa = min(kThreads / 32, (ga + 31) / 32), nwb = min(kThreads / 32, (gb + 31) / 32);
    int status = ST_RUNNING, inner = ST_RUNNING;
    float beta = (float)beta64;
    for (;;) {
        // ---- A: direction, A p, p.q
#pragma unroll
        for (int k = 0; k < NT; ++k) {
            float* p = P(k);
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                float4* pv = reinterpret_cast<float4*>(p + (2 * warp + y + 1) * kBX + 4 + 4 * lane);
                const unsigned cd = code[k] >> (16 * y), vd = valid[k] >> (4 * y);
                float4 o = *pv, z = r[k][y];
                z.x = tab_m[cd & 15u] * z.x;
                z.y = tab_m[cd >> 4 & 15u] * z.y;
                z.z = tab_m[cd >> 8 & 15u] * z.z;
                z.w = tab_m[cd >> 12 & 15u] * z.w;
                if (!first) {
                    z.x = fmaf(beta, o.x, z.x);
                    z.y = fmaf(beta, o.y, z.y);
                    z.z = fmaf(beta, o.z, z.z);
                    z.w = fmaf(beta, o.w, z.w);
                }
                // (beyond the grid's edge the halo values stay)
                if ((vd & 15u) == 15u) {
                    *pv = z;
                } else {
                    float* f = reinterpret_cast<float*>(pv);
                    if (vd & 1u) f[0] = z.x;
                    if (vd & 2u) f[1] = z.y;
                    if (vd & 4u) f[2] = z.z;
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (hsrc[k][h] >= 0) {
                    float& v = p[hpos[k][h]];
                    v = first ? zh[k][h] : fmaf(beta, v, zh[k][h]);
                }
        }
        first = false;
        __syncthreads();
        float acc[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) acc[k] = 0.f;
#pragma unroll
        for (int k = 0; k < NT; ++k) {
            float part = 0.f;
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const float* rc = P(k) + (2 * warp + y + 1) * kBX + 4 + 4 * lane;
                const float4 pc = *reinterpret_cast<const float4*>(rc);
                const float4 pu = *reinterpret_cast<const float4*>(rc - kBX);
                const float4 pd = *reinterpret_cast<const float4*>(rc + kBX);
                const float left = rc[-1], right = rc[4];
                const unsigned cd = code[k] >> (16 * y), vd = valid[k] >> (4 * y);
                float4 v;
                v.x = fmaf(ms, pd.x, fmaf(ms, pu.x, fmaf(ms, pc.y, fmaf(ms, left, tab_d[cd & 15u] * pc.x))));
                v.y = fmaf(ms, pd.y, fmaf(ms, pu.y, fmaf(ms, pc.z, fmaf(ms, pc.x, tab_d[cd >> 4 & 15u] * pc.y))));
                v.z = fmaf(ms, pd.z, fmaf(ms, pu.z, fmaf(ms, pc.w, fmaf(ms, pc.y, tab_d[cd >> 8 & 15u] * pc.z))));
                v.w = fmaf(ms, pd.w, fmaf(ms, pu.w, fmaf(ms, right, fmaf(ms, pc.z, tab_d[cd >> 12 & 15u] * pc.w))));
                if (vd & 1u) part = fmaf(pc.x, v.x, part);
                if (vd & 2u) part = fmaf(pc.y, v.y, part);
                if (vd & 4u) part = fmaf(pc.z, v.z, part);
                if (vd & 8u) part = fmaf(pc.w, v.w, part);
                q[k][y] = v;
            }
            add_to(acc, k, na, part);
        }
        warp_sums(acc, na, red[0]);
        __syncthreads();
        put_partial(red[0], warp, min(na, NT), partA);
        grid_arrive(S);
        arrived += nb;
        if (!grid_wait(S, gbase + arrived, stall)) return;
        if (warp < nwa) {
            const double s = warp_fold_n(strided_sum(partA, ga, tid), ga - 32 * warp);
            if (lane == 0) ws0[warp] = s;
        }
        __syncthreads();
        if (warp == 0) {
            double pq = ws0[0];
            for (int k = 1; k < nwa; ++k) pq = pq + ws0[k];
            const double al = rho / pq;
            if (lane == 0) {
                bc_stat = isnan(pq) ? (int)ST_NAN : (!(pq > 0.0) ? (int)ST_BREAKDOWN : (int)ST_RUNNING);
                bc_a = al;
                bc_f = (float)al;
            }
        }
        __syncthreads();
        if (bc_stat == ST_NAN) status = ST_NAN;
        if (bc_stat == ST_BREAKDOWN) inner = ST_BREAKDOWN;  // FP32 noise floor: refine and restart
        if (bc_stat != ST_RUNNING) break;
        alpha64 = bc_a;
        const float alpha = bc_f, malpha = -alpha;
        // ---- B: residual, z, border, r.z and r.r
        float az[NT], ar[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) az[k] = ar[k] = 0.f;
#pragma unroll
        for (int k = 0; k < NT; ++k) {
            const int t = tile_of(k);
            const int nc = min(kTW, a.nx - (t % a.tiles_x) * kTW), nr = min(kTH, a.ny - (t / a.tiles_x) * kTH);
            float* bo = border + (size_t)t * kHalo;
            float prz = 0.f, prr = 0.f;
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                float4 rv = r[k][y];
                rv.x = fmaf(malpha, q[k][y].x, rv.x);
                rv.y = fmaf(malpha, q[k][y].y, rv.y);
                rv.z = fmaf(malpha, q[k][y].z, rv.z);
                rv.w = fmaf(malpha, q[k][y].w, rv.w);
                r[k][y] = rv;
                const int row = 2 * warp + y;
                const unsigned cd = code[k] >> (16 * y), vd = valid[k] >> (4 * y);
                const float zs[4] = {tab_m[cd & 15u] * rv.x, tab_m[cd >> 4 & 15u] * rv.y, tab_m[cd >> 8 & 15u] * rv.z,
                                     tab_m[cd >> 12 & 15u] * rv.w};
                const float rs[4] = {rv.x, rv.y, rv.z, rv.w};
                if (valid[k] >> 31) {
                    const float s2 = fmaf(rv.w, rv.w, fmaf(rv.z, rv.z, fmaf(rv.y, rv.y, rv.x * rv.x)));
                    prr += s2;
                    prz = fmaf(tab_m[0], s2, prz);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (vd >> c & 1u) {
                            prz = fmaf(rs[c], zs[c], prz);
                            prr = fmaf(rs[c], rs[c], prr);
                        }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (!(vd >> c & 1u)) continue;
                    const int cc = 4 * lane + c;
                    if (row == 0) __stcg(bo + cc, zs[c]);
                    if (row == nr - 1) __stcg(bo + kTW + cc, zs[c]);
                    if (cc == 0) __stcg(bo + 2 * kTW + row, zs[c]);
                    if (cc == nc - 1) __stcg(bo + 2 * kTW + kTH + row, zs[c]);
                }
            }
            add_to(az, k, nbb, prz);
            add_to(ar, k, nbb, prr);
        }
        warp_sums(az, nbb, red[0]);
        warp_sums(ar, nbb, red[1]);
        __syncthreads();
        if (warp < kThreads / 64)
            put_partial(red[0], warp, min(nbb, NT), partB0);
        else
            put_partial(red[1], warp - kThreads / 64, min(nbb, NT), partB1);
        grid_arrive(S);
        arrived += nb;
#pragma unroll
        for (int k = 0; k < NT; ++k)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const float4 pc = *reinterpret_cast<const float4*>(P(k) + (2 * warp + y + 1) * kBX + 4 + 4 * lane);
                x[k][y][0] = df_add_f(x[k][y][0], alpha * pc.x);
                x[k][y][1] = df_add_f(x[k][y][1], alpha * pc.y);
                x[k][y][2] = df_add_f(x[k][y][2], alpha * pc.z);
                x[k][y][3] = df_add_f(x[k][y][3], alpha * pc.w);
            }
        if (!grid_wait(S, gbase + arrived)) return;
#pragma unroll
        for (int k = 0; k < NT; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (hsrc[k][h] >= 0) zh[k][h] = __ldcg(border + hsrc[k][h]);
        const int wr = 2 * nwb <= kThreads / 32 ? warp - nwb : warp;
        if (warp < nwb) {
            const double s = warp_fold_n(strided_sum(partB0, gb, tid), gb - 32 * warp);
            if (lane == 0) ws0[warp] = s;
        }
        if (wr >= 0 && wr < nwb) {
            const double s = warp_fold_n(strided_sum(partB1, gb, wr * 32 + lane), gb - 32 * wr);
            if (lane == 0) ws1[wr] = s;
        }
        __syncthreads();
        if (warp == 0) {
            double rz = ws0[0];
            for (int k = 1; k < nwb; ++k) rz = rz + ws0[k];
            const double be = rz / rho;
            if (lane == 0) {
                bc_a = be;
                bc_b = rz;
                bc_f = (float)be;
            }
        } else if (warp == 1) {
            double t = ws1[0];
            for (int k = 1; k < nwb; ++k) t = t + ws1[k];
            if (lane == 0) bc_c = t;
        }
        __syncthreads();
        beta64 = bc_a;
        beta = bc_f;
        rho_prev = rho;
        rho = bc_b;
        rr = bc_c;
        if (rr > rr0) rr0 = rr;
        ++it;
        ++iter;
        // reliable update when the recursive residual fell by delta since the
        // last one, or already looks converged
        if (isnan(rr))
            status = ST_NAN;
        else if (rr <= S->tau2 * rr0 || rr <= S->target2)
            inner = ST_CONVERGED;
        else if (iter >= max_iter)
            inner = ST_MAXIT;
        if (status != ST_RUNNING || inner != ST_RUNNING || it >= it_end) break;
    }
    float* pnew = (it & 1) ? a.pb : a.pa;
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const int t = tile_of(k), i0 = (t % a.tiles_x) * kTW, j0 = (t / a.tiles_x) * kTH;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const int row = 2 * warp + y, j = j0 + row;
            const float rs[4] = {r[k][y].x, r[k][y].y, r[k][y].z, r[k][y].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (!(valid[k] >> (4 * y + c) & 1u)) continue;
                const int i = i0 + 4 * lane + c;
                a.x[(size_t)j * a.xpitch + i] = x[k][y][c];
                a.r[(ptrdiff_t)j * a.pitch + i] = rs[c];
                pnew[(ptrdiff_t)j * a.pitch + i] = P(k)[(row + 1) * kBX + 4 + 4 * lane + c];
            }
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        S->inner_iter = it;
        S->iter = iter;
        S->restart = 0;
        S->alpha_in = alpha64;
        S->beta_in = beta64;
        S->rho_prev = rho_prev;
        S->rho_in = rho;
        S->rr_in = rr;
        S->rr_in0 = rr0;
        S->gbar = gbase + arrived;
        S->inner_status = inner;
        atomicCAS(&S->status, (int)ST_RUNNING, status);  // a block's timeout stays
    }
}

// --------------------------------------------------------------------------
// Mixed MG-PCG helpers.  z = V-cycle(r) is written to the owned cells of z32;
// along periodic axes its ghost ring is refreshed here (wall ghosts stay 0).
__global__ void k_z32_ghosts(float* z, int nx, int ny, int pitch, int per_x, int per_y) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (per_x && t < ny) {
        float* row = z + (ptrdiff_t)t * pitch;
        row[-1] = row[nx - 1];
        row[nx] = row[0];
    }
    if (per_y && t < nx) {
        z[-(ptrdiff_t)pitch + t] = z[(ptrdiff_t)(ny - 1) * pitch + t];
        z[(ptrdiff_t)ny * pitch + t] = z[t];
    }
}

// rho = r.z (FP32 per lane over a 64 x 16 unit, FP64 beyond).  After an
// inner iteration: beta = rho_new / rho.  After the residual was re-formed
// from the FP64 solution (S->refreshed): beta = rho_new / rho_prev, which
// keeps the search direction across a reliable update (ignored on a restart).
__global__ void __launch_bounds__(CF_RED_THREADS)
    k_mg_rz32(const float* r, const float* z, int nx, int ny, int pitch, int G, int U, double* part,
              SolverState* S) {
    if (!running(S)) return;
    const int lane = threadIdx.x & 31;
    const int unit = blockIdx.x * CF_RED_WARPS + (threadIdx.x >> 5);
    float arz = 0.f;
    if (unit < U) {
        const int g = unit % G, band = unit / G;
        const int c0 = g * CF_UNIT_COLS + 2 * lane;
        const int j0 = band * CF_BAND_ROWS;
        const int j1 = min(j0 + CF_BAND_ROWS, ny);
        for (int j = j0; j < j1; ++j)
            for (int s = 0; s < 2; ++s) {
                const int c = c0 + s;
                if (c >= nx) continue;
                const ptrdiff_t k = (ptrdiff_t)j * pitch + c;
                arz = fmaf(r[k], z[k], arz);
            }
    }
    double drz = warp_fold((double)arz);
    if (unit < U && lane == 0) part[unit] = drz;
    if (last_block_arrive(&S->ticket[7])) {
        double rz = final_tree(part, U);
        if (threadIdx.x == 0) {
            S->ticket[7] = 0;
            double den = S->refreshed ? S->rho_prev : S->rho_in;
            S->refreshed = 0;
            S->beta_in = den != 0.0 ? rz / den : 0.0;
            S->rho_in = rz;
            if (isnan(rz))
                S->status = ST_NAN;
            else if (!(rz > 0.0))
                S->inner_status = ST_BREAKDOWN;  // FP32 noise floor: refine and restart
        }
    }
}

// --------------------------------------------------------------------------
// host side

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// 2-D map over a ghosted FP32 vector's storage (pitch x (ny + 2) floats)
static int make_map(cf_ctx* c, CUtensorMap* m, float* base) {
    auto fn = encode_fn();
    if (!fn) return fail(c, CF_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    cuuint64_t dims[2] = {(cuuint64_t)c->p32, (cuuint64_t)(c->ph.ny + 2)};
    cuuint64_t strides[1] = {(cuuint64_t)c->p32 * sizeof(float)};
    cuuint32_t box[2] = {(cuuint32_t)kBX, (cuuint32_t)kBY};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(c, CF_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return CF_OK;
}

static int pcg32_setup(cf_ctx* c);

int cg32_setup(cf_ctx* c) {
    int rc = make_map(c, &c->map_r, c->r32b);
    if (!rc) rc = make_map(c, &c->map_pa, c->pa32b);
    if (!rc) rc = make_map(c, &c->map_pb, c->pb32b);
    if (rc) return rc;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    c->tiles_x = (c->ph.nx + kTW - 1) / kTW;
    c->tiles = c->tiles_x * ((c->ph.ny + kTH - 1) / kTH);
    rc = cuda_check(c, cudaFuncSetAttribute(k_tma_dir_matvec32<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            kStages * 2 * kSlot + 128),
                    "smem attribute");
    if (!rc)
        rc = cuda_check(c, cudaFuncSetAttribute(k_tma_dir_matvec32<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                kStages * 2 * kSlot + 128),
                        "smem attribute");
    if (!rc)
        rc = cuda_check(c, cudaFuncSetAttribute(k_tma_update32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                kStages * 2 * kSlot + 128),
                        "smem attribute");
    // persistent grids: as many CTAs as fit on the GPU at once
    int occ1 = 0, occ2 = 0;
    if (!rc)
        rc = cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ1, k_tma_dir_matvec32<false>, kThreads,
                                                                         kStages * 2 * kSlot + 128),
                        "occupancy");
    if (!rc)
        rc = cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, k_tma_update32, kThreads,
                                                                         kStages * 2 * kSlot + 128),
                        "occupancy");
    if (rc) return rc;
    occ1 = std::clamp(occ1, 1, kCtas1);
    occ2 = std::clamp(occ2, 1, kCtas2);
    c->cta32 = c->tiles < occ1 * sms ? c->tiles : occ1 * sms;
    c->cta32b = c->tiles < occ2 * sms ? c->tiles : occ2 * sms;
    return pcg32_setup(c);
}

template <int NT>
static constexpr size_t pcg32_smem() { return sizeof(float) * NT * kBY * kBX; }
template <int NT>
static bool pcg32_fits(const cf_ctx* c) {
    return all_fit(k_pcg32<NT>, c->pcg_blocks, kThreads, pcg32_smem<NT>(), c->sms);
}

// Tiles per block of the on-chip inner solve (0: the grid does not fit) and the
// border buffer.  Up to four tiles per SM; more than one of the launch-per-phase
// kernels' block would walk in turn only where those fill every SM alike, so that
// one block here holds them all.
static int pcg32_setup(cf_ctx* c) {
    c->pcg_nu = 0;
    const int per = (c->tiles + c->sms - 1) / c->sms;
    if (per > kMaxTiles) return CF_OK;
    if ((c->cta32 < c->tiles && c->cta32 % c->sms) || (c->cta32b < c->tiles && c->cta32b % c->sms)) return CF_OK;
    const int nt = per <= 1 ? 1 : (per <= 2 ? 2 : kMaxTiles);
    c->pcg_blocks = std::min(c->tiles, c->sms);
    const bool fits = nt == 1 ? pcg32_fits<1>(c) : (nt == 2 ? pcg32_fits<2>(c) : pcg32_fits<kMaxTiles>(c));
    if (!fits) return CF_OK;
    void* p = nullptr;
    const size_t bytes = sizeof(float) * kHalo * (size_t)c->tiles;
    if (cudaMalloc(&p, bytes) != cudaSuccess) return fail(c, CF_ERR_NOMEM, "cudaMalloc of %zu bytes failed", bytes);
    c->allocs.push_back(p);
    c->pcg_border = p;
    c->pcg_nu = nt;
    return CF_OK;
}

// z32 (ghosted, zero) and its tensor map, for the mixed MG-PCG
int cg32_mg_setup(cf_ctx* c) {
    if (c->z32b) return CF_OK;
    size_t n32 = (size_t)c->p32 * (c->ph.ny + 2);
    cudaError_t e = cudaMalloc(&c->z32b, n32 * sizeof(float));
    if (e != cudaSuccess) return fail(c, CF_ERR_NOMEM, "z32: cudaMalloc failed");
    c->allocs.push_back(c->z32b);
    int rc = cuda_check(c, cudaMemsetAsync(c->z32b, 0, n32 * sizeof(float), c->stream), "z32 memset");
    c->z32.a = c->z32b + c->p32 + 4;
    c->z32.pitch = c->p32;
    if (!rc) rc = make_map(c, &c->map_z, c->z32b);
    return rc;
}

static Cg32T cg32_args(cf_ctx* c, const Stencil& st) {
    Cg32T a{};
    a.nx = c->ph.nx;
    a.ny = c->ph.ny;
    a.per_x = c->ph.per_x;
    a.per_y = c->ph.per_y;
    a.tiles_x = c->tiles_x;
    a.tiles = c->tiles;
    a.pitch = c->p32;
    a.st = st;
    a.x = reinterpret_cast<float2*>(c->x.a);
    a.xpitch = c->vpitch;
    a.r = c->r32.a;
    a.pa = c->pa32.a;
    a.pb = c->pb32.a;
    a.part0 = c->partials;
    a.part1 = c->partials + c->n_units;
    a.S = c->S;
    return a;
}

void cg32_launch_iteration(cf_ctx* c, const Stencil& st) {
    Cg32T a = cg32_args(c, st);
    k_tma_dir_matvec32<false><<<c->cta32, kThreads, kStages * 2 * kSlot + 128, c->stream>>>(c->map_r, c->map_pa, c->map_pb, a);
    k_tma_update32<<<c->cta32b, kThreads, kStages * 2 * kSlot + 128, c->stream>>>(c->map_r, c->map_pa, c->map_pb,
                                                                            a);
}

// up to iters inner iterations in one launch (context with pcg_nu > 0)
cudaError_t pcg32_launch(cf_ctx* c, const Stencil& st, int iters) {
    const Cg32T a = cg32_args(c, st);
    float* border = static_cast<float*>(c->pcg_border);
    const int n = c->pcg_blocks;
    switch (c->pcg_nu) {
        case 1: return launch_all(k_pcg32<1>, n, kThreads, pcg32_smem<1>(), c->stream, a, border, c->cta32, c->cta32b, iters);
        case 2: return launch_all(k_pcg32<2>, n, kThreads, pcg32_smem<2>(), c->stream, a, border, c->cta32, c->cta32b, iters);
        default:
            return launch_all(k_pcg32<kMaxTiles>, n, kThreads, pcg32_smem<kMaxTiles>(), c->stream, a, border, c->cta32,
                              c->cta32b, iters);
    }
}

// z = V-cycle(r32), its periodic ghosts, rho = r.z; returns kernels launched
int cg32_mg_precondition(cf_ctx* c, double scale) {
    bool done = false;
    int n = mg_vcycle(c, scale, &done);
    if (done) return n;  // r.z, the scalars and z's ghosts came with the finest post-smoothing
    if (c->ph.per_x || c->ph.per_y) {
        int m = c->ph.nx > c->ph.ny ? c->ph.nx : c->ph.ny;
        k_z32_ghosts<<<(m + 255) / 256, 256, 0, c->stream>>>(c->z32.a, c->ph.nx, c->ph.ny, c->p32, c->ph.per_x,
                                                             c->ph.per_y);
        n += 1;
    }
    k_mg_rz32<<<(c->n_units + CF_RED_WARPS - 1) / CF_RED_WARPS, CF_RED_THREADS, 0, c->stream>>>(
        c->r32.a, c->z32.a, c->ph.nx, c->ph.ny, c->p32, c->G, c->n_units, c->partials, c->S);
    return n + 1;
}

// K1 on z (M^-1 = 1) and K2 of one MG-PCG inner iteration.  When every
// iteration ends with a reliable update (c->x_only), K2 reduces to the x
// update, which the fused reliable update does (k_outer_resid<true>), so K1
// runs alone.
void cg32_launch_pair_mg(cf_ctx* c, const Stencil& st) {
    Stencil stz = st;
    for (int b = 0; b < 16; ++b) stz.minv32[b] = 1.0f;
    Cg32T a = cg32_args(c, stz);
    a.mg = 1;
    k_tma_dir_matvec32<true><<<c->cta32, kThreads, kStages * 2 * kSlot + 128, c->stream>>>(c->map_z, c->map_pa, c->map_pb, a);
    if (!c->x_only) {
        k_tma_update32<<<c->cta32b, kThreads, kStages * 2 * kSlot + 128, c->stream>>>(c->map_r, c->map_pa, c->map_pb,
                                                                                a);
    }
}

}  // namespace cf
