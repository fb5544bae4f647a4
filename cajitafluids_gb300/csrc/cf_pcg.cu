// Jacobi-PCG with the whole solve on chip, for grids whose solver vectors fit
// the SMs' shared memory.
//
// As launches (cf_project.cu: a block per unit of 64 x 16 cells) an iteration is two
// kernels, each of which starts, reads its vectors, is folded by its last block and
// drains: 23 us at 256^2, of which the FP64 work (an SM executes one FP64 warp
// instruction per sub-partition every 64 cycles) is two.  Here one cooperative launch
// runs many iterations: a block owns NU units (r, p with its
// halo and A p / z in shared memory, x in registers), the grid meets at two
// barriers per iteration, and every block folds the unit partials itself.
//
//   A  p <- z + beta p (own cells and halo); q <- A p; unit partials of p.q
//   -- barrier, fold, alpha
//   B  r <- r - alpha q; z <- M^-1 r; border z published; unit partials of
//      r.z and r.r; x <- x + alpha p between arriving and waiting
//   -- barrier, fold, beta, convergence
//
// A unit's partial is the canonical one (cf_internal.cuh): lane l adds its two
// columns row by row with fused multiply-adds, one warp per unit and sum, from
// the products' factors staged in shared memory; the cells themselves are
// computed by the whole block.  Every cell value and every
// sum is formed by the same operations in the same order as by
// k_cg_dir_matvec64 and k_cg_update64, so the results are the same bits.
//
// What bounds it: with one or two units per SM the serial lane sums (32
// dependent FMAs of 64 cycles, 1 us each phase), the two grid barriers (about
// 1.2 us each) and the divisions; at seven units per SM the FP64 pipe (10
// operations per cell and iteration: 18 of 31 us).  Measured on GB300, time of
// one iteration, launches (with eight units to a block, as they were then) and this:
// 64^2 39.9 -> 9.7 us, 256^2 49.6 -> 10.4 us, 1024^2 53.8 -> 31.2 us; 1072^2, with a unit
// to a block, 44.4 -> 34.7 us.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "cf_grid.cuh"
#include "cf_mul64.cuh"

namespace cf {

// threads per block: the lane sums and folds of one or two units keep few
// warps busy; more have the cells to keep 16 warps issuing
template <int NU>
struct PcThreads {
    static constexpr int value = NU <= 2 ? 256 : 512;
};
// Plain products: more than two units per block are bound by the FP64 pipe, and
// products on the integer pipes run beside it (1024^2: 33.2 -> 31.1 us an iteration);
// one or two units wait for results, which the hardware product returns sooner
// (a 256^2 step: 10.2 ms against 10.4 with integer products).
template <int NU>
__device__ __forceinline__ double pcg_mul(double a, double b) {
    return NU <= 2 ? a * b : mul64i(a, b);
}
constexpr int PC_PW = UNIT_PW, PC_P = UNIT_P, PC_CELLS = UNIT_CELLS, PC_BORDER = UNIT_BORDER;
constexpr int PC_UNIT = PC_P + 2 * PC_CELLS;  // doubles per unit: p with its halo, r, q / z
constexpr int PC_MAX_UNITS = 8;  // units per block: 207 KB of the 227 KB of shared memory a block may have
struct Pcg64 {
    int nx, ny, per_x, per_y, G, U, pitch;
    Stencil st;
    double *x, *r, *pa, *pb;
    double* border;                 // PC_BORDER values of z per unit
    double *partA, *partB0, *partB1;  // unit partials: p.q; r.z, r.r
    SolverState* S;
    int iters;                      // iterations of this launch at most
};

// halo cell t of a unit in the border its owner publishes (first row, last row,
// first column, last column): the owner's last row lies below the unit, its
// first row above, its last column west, its first column east
__device__ __forceinline__ int border_of(int t) {
    return t < CF_UNIT_COLS                      ? CF_UNIT_COLS + t
           : t < 2 * CF_UNIT_COLS                ? t - CF_UNIT_COLS
           : t < 2 * CF_UNIT_COLS + CF_BAND_ROWS ? t + CF_BAND_ROWS
                                                 : t - CF_BAND_ROWS;
}

template <int NU>
__global__ void __launch_bounds__(PcThreads<NU>::value, 1) k_pcg64(Pcg64 a) {
    constexpr int PC_THREADS = PcThreads<NU>::value, PC_CPT = PC_CELLS / PC_THREADS;
    extern __shared__ __align__(16) double pc_smem[];
    __shared__ double tab_d[16], tab_m[16];
    __shared__ double ws0[CF_RED_WARPS], ws1[CF_RED_WARPS];
    __shared__ double bc_val;
    __shared__ int bc_stat;
    SolverState* S = a.S;
    if (*(volatile int*)&S->status != ST_RUNNING) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int it = S->iter;
    const int it_end = it + a.iters, max_iter = S->max_iter;
    double beta = S->beta, rho = S->rho, rr = S->rr, alpha = S->alpha;
    const bool stall = S->test_stall != 0 && blockIdx.x == 0;
    const unsigned gbase = S->gbar;
    unsigned arrived = 0;
    if (tid < 16) {
        tab_d[tid] = a.st.diag[tid];
        tab_m[tid] = a.st.minv[tid];
    }
    __syncthreads();
    const double ms = a.st.ms;
    auto unit_of = [&](int k) { return (int)blockIdx.x + k * (int)gridDim.x; };
    auto P = [&](int k) { return pc_smem + k * PC_UNIT; };
    auto R = [&](int k) { return pc_smem + k * PC_UNIT + PC_P; };
    auto Q = [&](int k) { return pc_smem + k * PC_UNIT + PC_P + PC_CELLS; };

    // Thread t owns cells t, t + PC_THREADS, ... of each unit (64 to a row: row
    // t / 64 + m PC_THREADS / 64, column t % 64) and, below PC_BORDER, one halo value.
    // code[k]: 4 wall-adjacency bits per cell, then a valid bit per cell.
    const int col = tid & (CF_UNIT_COLS - 1), row0 = tid / CF_UNIT_COLS;
    double xr[NU][PC_CPT];
    unsigned code[NU];
    int hsrc[NU], hpos[NU];  // border value this thread reads (-1: none, a wall), and its place in p
    double zh[NU];
    const double* pold = (it & 1) ? a.pb : a.pa;
#pragma unroll
    for (int k = 0; k < NU; ++k) {
        const int u = unit_of(k);
        code[k] = 0;
        hsrc[k] = -1;
        hpos[k] = 0;
        zh[k] = 0.0;
        if (u >= a.U) continue;
        const int g = u % a.G, band = u / a.G;
        const int c0 = g * CF_UNIT_COLS, j0 = band * CF_BAND_ROWS;
        const int nc = min(CF_UNIT_COLS, a.nx - c0), nr = min(CF_BAND_ROWS, a.ny - j0);
        double *p = P(k), *r = R(k), *q = Q(k);
        for (int i = tid; i < PC_P; i += PC_THREADS) p[i] = 0.0;
        __syncthreads();
#pragma unroll
        for (int m = 0; m < PC_CPT; ++m) {
            const int row = row0 + m * (PC_THREADS / CF_UNIT_COLS), cell = row * CF_UNIT_COLS + col;
            double rv = 0.0, z = 0.0;
            xr[k][m] = 0.0;
            if (col < nc && row < nr) {
                const int eb = edge_bits(c0 + col, j0 + row, a.nx, a.ny, a.per_x, a.per_y);
                code[k] |= (unsigned)eb << (4 * m) | 1u << (16 + m);
                const size_t o = (size_t)(j0 + row) * a.pitch + c0 + col;
                rv = a.r[o];
                z = pcg_mul<NU>(tab_m[eb], rv);
                xr[k][m] = a.x[o];
                if (it > 0) p[(row + 1) * PC_PW + col + 1] = pold[o];
            }
            r[cell] = rv;
            q[cell] = z;
        }
        // halo: row below, row above, column west, column east of the unit's
        // cells in the grid (wrapped along a periodic axis, 0 beyond a wall)
        if (tid < PC_BORDER) {
            int gc, gj, pos;
            const bool in = unit_halo(UnitPos{c0, j0, nc, nr}, tid, gc, gj, pos);
            const int off = border_of(tid);
            const int wc = wrap_index(gc, a.nx, a.per_x), wj = wrap_index(gj, a.ny, a.per_y);
            if (in && wc >= 0 && wj >= 0) {
                const int ou = (wj / CF_BAND_ROWS) * a.G + wc / CF_UNIT_COLS;
                hsrc[k] = ou * PC_BORDER + off;
                hpos[k] = pos;
                const size_t o = (size_t)wj * a.pitch + wc;
                zh[k] = tab_m[edge_bits(wc, wj, a.nx, a.ny, a.per_x, a.per_y)] * a.r[o];
                if (it > 0) p[pos] = pold[o];
            }
        }
        __syncthreads();
    }
    int status = ST_RUNNING;
    const int nw = min(CF_RED_WARPS, (a.U + 31) / 32);  // warps whose strided sums are not empty
    for (;;) {
        // ---- A: direction, A p, p.q
        const bool first = it == 0;
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            if (unit_of(k) >= a.U) break;
            double *p = P(k), *q = Q(k);
#pragma unroll
            for (int m = 0; m < PC_CPT; ++m) {
                const int row = row0 + m * (PC_THREADS / CF_UNIT_COLS);
                if (code[k] >> (16 + m) & 1u) {
                    const double z = q[row * CF_UNIT_COLS + col];
                    double& pv = p[(row + 1) * PC_PW + col + 1];
                    pv = first ? z : fma(beta, pv, z);
                }
            }
            if (hsrc[k] >= 0) p[hpos[k]] = first ? zh[k] : fma(beta, p[hpos[k]], zh[k]);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            if (unit_of(k) >= a.U) break;
            const double* p = P(k);
            double* q = Q(k);
#pragma unroll
            for (int m = 0; m < PC_CPT; ++m) {
                const int row = row0 + m * (PC_THREADS / CF_UNIT_COLS);
                const double* c = p + (row + 1) * PC_PW + col + 1;
                double qv = 0.0;
                if (code[k] >> (16 + m) & 1u) {
                    qv = pcg_mul<NU>(tab_d[code[k] >> (4 * m) & 15u], c[0]);
                    qv = fma(ms, c[-1], qv);
                    qv = fma(ms, c[1], qv);
                    qv = fma(ms, c[-PC_PW], qv);
                    qv = fma(ms, c[PC_PW], qv);
                }
                q[row * CF_UNIT_COLS + col] = qv;
            }
        }
        __syncthreads();
        if (warp < NU && unit_of(warp) < a.U) {
            const double s = unit_dot(P(warp) + PC_PW + 1, PC_PW, Q(warp), CF_UNIT_COLS, lane);
            if (lane == 0) __stcg(a.partA + unit_of(warp), s);
        }
        grid_arrive(S);
        arrived += gridDim.x;
        if (!grid_wait(S, gbase + arrived, stall)) return;
        if (warp < nw) {
            const double s = warp_fold_n(strided_sum(a.partA, a.U, tid), a.U - 32 * warp);
            if (lane == 0) ws0[warp] = s;
        }
        __syncthreads();
        if (warp == 0) {
            double pq = ws0[0];
            for (int k = 1; k < nw; ++k) pq = pq + ws0[k];
            const double al = rho / pq;
            if (lane == 0) {
                bc_stat = !(pq > 0.0) ? (isnan(pq) ? (int)ST_NAN : (int)ST_BREAKDOWN) : (int)ST_RUNNING;
                bc_val = al;
            }
        }
        __syncthreads();
        status = bc_stat;
        if (status != ST_RUNNING) break;
        alpha = bc_val;
        // ---- B: residual, z, border, r.z and r.r
        const double malpha = -alpha;
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const int u = unit_of(k);
            if (u >= a.U) break;
            double *r = R(k), *q = Q(k);
            double* bo = a.border + (size_t)u * PC_BORDER;
            const int nc = min(CF_UNIT_COLS, a.nx - (u % a.G) * CF_UNIT_COLS);
            const int nr = min(CF_BAND_ROWS, a.ny - (u / a.G) * CF_BAND_ROWS);
#pragma unroll
            for (int m = 0; m < PC_CPT; ++m) {
                const int row = row0 + m * (PC_THREADS / CF_UNIT_COLS), cell = row * CF_UNIT_COLS + col;
                if (!(code[k] >> (16 + m) & 1u)) continue;
                const double rv = fma(malpha, q[cell], r[cell]);
                const double z = pcg_mul<NU>(tab_m[code[k] >> (4 * m) & 15u], rv);
                r[cell] = rv;
                q[cell] = z;
                if (row == 0) __stcg(bo + col, z);
                if (row == nr - 1) __stcg(bo + CF_UNIT_COLS + col, z);
                if (col == 0) __stcg(bo + 2 * CF_UNIT_COLS + row, z);
                if (col == nc - 1) __stcg(bo + 2 * CF_UNIT_COLS + CF_BAND_ROWS + row, z);
            }
        }
        __syncthreads();
        for (int c = warp; c < 2 * NU; c += PC_THREADS / 32) {
            const int k = c >> 1, u = unit_of(k);
            if (u >= a.U) break;
            const double s = unit_dot(R(k), CF_UNIT_COLS, (c & 1) ? R(k) : Q(k), CF_UNIT_COLS, lane);
            if (lane == 0) __stcg(((c & 1) ? a.partB1 : a.partB0) + u, s);
        }
        grid_arrive(S);
        arrived += gridDim.x;
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            if (unit_of(k) >= a.U) break;
            const double* p = P(k);
#pragma unroll
            for (int m = 0; m < PC_CPT; ++m) {
                const int row = row0 + m * (PC_THREADS / CF_UNIT_COLS);
                if (code[k] >> (16 + m) & 1u) xr[k][m] = fma(alpha, p[(row + 1) * PC_PW + col + 1], xr[k][m]);
            }
        }
        if (!grid_wait(S, gbase + arrived)) return;
#pragma unroll
        for (int k = 0; k < NU; ++k)
            if (hsrc[k] >= 0) zh[k] = __ldcg(a.border + hsrc[k]);
        // r.z by warps 0 .. nw - 1, r.r by the next nw (or the same where the
        // block has too few)
        const int wr = 2 * nw <= PC_THREADS / 32 ? warp - nw : warp;
        if (warp < nw) {
            const double s = warp_fold_n(strided_sum(a.partB0, a.U, tid), a.U - 32 * warp);
            if (lane == 0) ws0[warp] = s;
        }
        if (wr >= 0 && wr < nw) {
            const double s = warp_fold_n(strided_sum(a.partB1, a.U, wr * 32 + lane), a.U - 32 * wr);
            if (lane == 0) ws1[wr] = s;
        }
        __syncthreads();
        if (warp == 0) {
            double rz = ws0[0];
            for (int k = 1; k < nw; ++k) rz = rz + ws0[k];
            const double be = rz / rho;
            if (lane == 0) {
                bc_val = be;
                ws0[0] = rz;
            }
        } else if (warp == 1) {
            double t = ws1[0];
            for (int k = 1; k < nw; ++k) t = t + ws1[k];
            int st = ST_RUNNING;
            if (isnan(t))
                st = ST_NAN;
            else if (t <= S->tol2 * S->bb || (S->use_abs && t * S->area <= S->abs2))
                st = ST_CONVERGED;
            else if (it + 1 >= max_iter)
                st = ST_MAXIT;
            if (lane == 0) {
                bc_stat = st;
                ws1[0] = t;
            }
        }
        __syncthreads();
        beta = bc_val;
        rho = ws0[0];
        rr = ws1[0];
        status = bc_stat;
        ++it;
        if (status != ST_RUNNING || it >= it_end) break;
        __syncthreads();  // ws0 and ws1 are read above and written again below
    }
    // x always; r and p for the next launch of the same solve
    double* pnew = (it & 1) ? a.pb : a.pa;
#pragma unroll
    for (int k = 0; k < NU; ++k) {
        const int u = unit_of(k);
        if (u >= a.U) break;
        const int c0 = (u % a.G) * CF_UNIT_COLS, j0 = (u / a.G) * CF_BAND_ROWS;
#pragma unroll
        for (int m = 0; m < PC_CPT; ++m) {
            const int row = row0 + m * (PC_THREADS / CF_UNIT_COLS), cell = row * CF_UNIT_COLS + col;
            if (!(code[k] >> (16 + m) & 1u)) continue;
            const size_t o = (size_t)(j0 + row) * a.pitch + c0 + col;
            a.x[o] = xr[k][m];
            a.r[o] = R(k)[cell];
            pnew[o] = P(k)[(row + 1) * PC_PW + col + 1];
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        S->iter = it;
        S->alpha = alpha;
        S->beta = beta;
        S->rho = rho;
        S->rr = rr;
        S->gbar = gbase + arrived;
        atomicCAS(&S->status, (int)ST_RUNNING, status);  // a block's timeout stays
    }
}

// --------------------------------------------------------------------------
// host side

template <int NU>
static constexpr size_t pcg64_smem() { return sizeof(double) * PC_UNIT * NU; }
template <int NU>
static bool pcg64_fits(const cf_ctx* c) {
    return all_fit(k_pcg64<NU>, c->pcg_blocks, PcThreads<NU>::value, pcg64_smem<NU>(), c->sms);
}

// Units per block of the on-chip solve (0: the grid does not fit), and the
// border buffer.  A block takes as few units as the SMs allow, up to the eight whose
// vectors shared memory holds (1216 units on 152 SMs); the solve is faster than the
// launches at every such size (above).  The loops over a block's units are unrolled for
// one, two, four, seven or eight: with eight where seven do, 1024^2 takes 0.4 % longer.
int pcg64_setup(cf_ctx* c) {
    c->pcg_nu = 0;
    const int per = (c->n_units + c->sms - 1) / c->sms;
    if (per > PC_MAX_UNITS) return CF_OK;
    const int nu = per <= 2 ? per : (per <= 4 ? 4 : (per <= 7 ? 7 : PC_MAX_UNITS));
    c->pcg_blocks = std::min(c->n_units, c->sms);
    const bool fits = nu == 1   ? pcg64_fits<1>(c)
                      : nu == 2 ? pcg64_fits<2>(c)
                      : nu == 4 ? pcg64_fits<4>(c)
                      : nu == 7 ? pcg64_fits<7>(c)
                                : pcg64_fits<PC_MAX_UNITS>(c);
    if (!fits) return CF_OK;
    void* p = nullptr;
    const size_t bytes = sizeof(double) * PC_BORDER * (size_t)c->n_units;
    if (cudaMalloc(&p, bytes) != cudaSuccess) return fail(c, CF_ERR_NOMEM, "cudaMalloc of %zu bytes failed", bytes);
    c->allocs.push_back(p);
    c->pcg_border = p;
    c->pcg_nu = nu;
    return CF_OK;
}

// up to iters Jacobi-PCG iterations in one launch (context with pcg_nu > 0)
cudaError_t pcg64_launch(cf_ctx* c, const Stencil& st, int iters) {
    Pcg64 a{};
    a.nx = c->ph.nx;
    a.ny = c->ph.ny;
    a.per_x = c->ph.per_x;
    a.per_y = c->ph.per_y;
    a.G = c->G;
    a.U = c->n_units;
    a.pitch = c->vpitch;
    a.st = st;
    a.x = c->x.a;
    a.r = c->r.a;
    a.pa = c->pa.a;
    a.pb = c->pb.a;
    a.border = static_cast<double*>(c->pcg_border);
    a.partA = c->partials;
    a.partB0 = c->partials + c->n_units;
    a.partB1 = c->partials + 2 * (size_t)c->n_units;
    a.S = c->S;
    a.iters = iters;
    const int n = c->pcg_blocks;
    switch (c->pcg_nu) {
        case 1: return launch_all(k_pcg64<1>, n, PcThreads<1>::value, pcg64_smem<1>(), c->stream, a);
        case 2: return launch_all(k_pcg64<2>, n, PcThreads<2>::value, pcg64_smem<2>(), c->stream, a);
        case 4: return launch_all(k_pcg64<4>, n, PcThreads<4>::value, pcg64_smem<4>(), c->stream, a);
        case 7: return launch_all(k_pcg64<7>, n, PcThreads<7>::value, pcg64_smem<7>(), c->stream, a);
        default:
            return launch_all(k_pcg64<PC_MAX_UNITS>, n, PcThreads<PC_MAX_UNITS>::value, pcg64_smem<PC_MAX_UNITS>(), c->stream, a);
    }
}

}  // namespace cf
