// One multigrid level per launch with a row per warp, for the levels between the
// cluster launch (cf_mgc.cuh) and the register strips (included by cf_mg.cu; the
// same values cell for cell).
//
// A block takes a window of 128 columns (small FP64 levels: 64) x up to 32 rows: warp
// w holds row w in registers, lane l its columns 4l .. 4l + 3; west and east neighbours are the
// lane's own or come by shuffle, the rows above and below through shared memory,
// where a row keeps its red and its black cells apart.  The window's edge is
// recomputed by its neighbours (pre-smoothing: 8 | 112 | 8 columns, or 6 | 52 | 6,
// and 5 rows above and below those kept; post-smoothing: 4 | 120 | 4, 4 | 56 | 4 and 4).  Columns beyond
// a wall carry a reciprocal diagonal of zero, so they stay zero without a test;
// columns and rows across a periodic wrap are computed as copies.  Blocks walk the
// windows; the next window's right-hand side is fetched while one is worked on.
//
// Why: tiles of 32 x 16 in shared memory read five neighbours per update there
// with a stride of two (two wavefronts each) and computed 2.1 cells per cell kept.
// us, tiles -> rows: FP32 1024^2 pre 17.8 -> 10.6, post with r.z 35.6 -> 18.2;
// FP32 512^2 9.2 -> 4.7 and 8.7 -> 5.6; FP64 (bound by the FP64 pipe) 512^2 30.2
// -> 18.0 and 37.3 -> 17.3, 256^2 11.4 -> 8.0 and 10.8 -> 7.7.  The height of a
// window is chosen per level (mt_grid): 32 rows for all left 120 and 36 blocks on
// the FP64 levels above, 22.6 us each.
#pragma once

constexpr int MT_THREADS = 1024;
constexpr int MT_ROWS = 32;                   // most rows of a window (a warp each)
// Columns of a window, CPL (4, or 2 in FP64) to a lane, and those not kept at either
// side (at least six and four; the coarse columns under a lane are its own)
template <int CPL>
struct MtCols {
    static constexpr int all = 32 * CPL;
    static constexpr int pre_halo = CPL == 4 ? 8 : 6, post_halo = 4;
    static constexpr int pre = all - 2 * pre_halo, post = all - 2 * post_halo;
};
constexpr int MT_PRE_HALO = 10, MT_POST_HALO = 8;     // rows of a window not kept
constexpr int MT_RZ_ROWS = 16 + MT_POST_HALO;         // rows of a post-smoothing window that forms r.z

template <typename T, int CPL>
struct MtRow {
    static constexpr int HC = CPL / 2, COLS = MtCols<CPL>::all;
    int lane, g, c0;              // row and the lane's first column (not wrapped)
    bool live;                    // the row is in the grid (or wraps into it)
    T* row;                       // this row in shared memory, at the lane's cells
    const T *south, *north;
    T id[CPL];                    // 1 / diagonal per column, 0 beyond a wall
    T x[CPL], b[CPL];

    __device__ __forceinline__ T west() const { return __shfl_up_sync(0xffffffffu, x[CPL - 1], 1); }
    __device__ __forceinline__ T east() const { return __shfl_down_sync(0xffffffffu, x[0], 1); }
    __device__ __forceinline__ void store(int color) const {
        T v[HC];
        const bool odd = (g + color) & 1;
#pragma unroll
        for (int i = 0; i < HC; ++i) v[i] = odd ? x[2 * i + 1] : x[2 * i];
        mc_st<HC>(row + color * (COLS / 2), v);
    }
    // half sweep of one colour; the rows above and below hold the other one
    template <bool FIRST>
    __device__ __forceinline__ void half(int color, T scale) {
        T s[HC], n[HC], v[HC];
        if (!FIRST) {
            mc_ld<HC>(s, south + (1 - color) * (COLS / 2));
            mc_ld<HC>(n, north + (1 - color) * (COLS / 2));
        }
        if (((g + color) & 1) == 0) {
            const T w = FIRST ? T(0) : west();
#pragma unroll
            for (int i = 0; i < HC; ++i) {
                T t = b[2 * i];
                if (!FIRST) {
                    t = (i == 0 ? w : x[(2 * i + CPL - 1) % CPL]) + x[2 * i + 1];
                    t = t + s[i];
                    t = t + n[i];
                    t = mg_fma(scale, t, b[2 * i]);
                }
                v[i] = x[2 * i] = t * id[2 * i];
            }
        } else {
            const T e = FIRST ? T(0) : east();
#pragma unroll
            for (int i = 0; i < HC; ++i) {
                T t = b[2 * i + 1];
                if (!FIRST) {
                    t = x[2 * i] + (i == HC - 1 ? e : x[(2 * i + 2) % CPL]);
                    t = t + s[i];
                    t = t + n[i];
                    t = mg_fma(scale, t, b[2 * i + 1]);
                }
                v[i] = x[2 * i + 1] = t * id[2 * i + 1];
            }
        }
        mc_st<HC>(row + color * (COLS / 2), v);
    }
};

// a lane's values of a row of the level (a: row 0) from column c on, wrapped along a
// periodic axis and zero beyond a wall; inside: all in the grid
template <int CPL, typename T>
__device__ __forceinline__ void mt_load(T* v, const T* a, int pitch, int nx, int gw, int c, bool inside, int per_x) {
    const T* row = a + (size_t)gw * pitch;
    if (inside) {
        mc_ld<CPL>(v, row + c);
    } else {
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            const int i = mg_dom(c + k, nx, per_x);
            v[k] = i >= 0 ? row[i] : T(0);
        }
    }
}

// the wall-adjacency bits of the lane's columns (4 bits each; the row's bits
// included)
template <int CPL>
__device__ __forceinline__ unsigned mt_bits(const MgBc& p, int nx, int ny, int g, int c0) {
    unsigned rb = p.per_y ? 0u : (g == 0 ? 4u : 0u) | (g == ny - 1 ? 8u : 0u), code = 0;
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        const int c = c0 + k;
        code |= (rb | (p.per_x ? 0u : (c == 0 ? 1u : 0u) | (c == nx - 1 ? 2u : 0u))) << (4 * k);
    }
    return code;
}

template <typename T, int CPL>
__device__ __forceinline__ void mt_open(MtRow<T, CPL>& r, const MgLev<T>& F, const MgBc& p, const T* tab, T* rows, const T* zero,
                                        unsigned& code) {
    const int warp = threadIdx.x >> 5;
    constexpr int HC = CPL / 2, COLS = MtCols<CPL>::all;
    r.row = rows + warp * COLS + r.lane * HC;
    const bool ws = !p.per_y && r.g == 0, wn = !p.per_y && r.g == F.ny - 1;
    r.south = ws ? zero + r.lane * HC : r.row - COLS;
    r.north = wn ? zero + r.lane * HC : r.row + COLS;
    code = mt_bits<CPL>(p, F.nx, F.ny, r.g, r.c0);
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        const bool in = p.per_x || (r.c0 + k >= 0 && r.c0 + k < F.nx);
        r.id[k] = in ? tab[16 + (code >> (4 * k) & 15u)] : T(0);
    }
}

// x = 0, (red, black) x 2, x to the level's r array, r = b - A x, b_coarse = R r
template <typename T, int CPL>
__global__ void __launch_bounds__(MT_THREADS, 1) k_mg_pre_rows(const __grid_constant__ MgLev<T> F, T* cb, int cpitch, MgBc p,
                                                               SolverState* S, int inner, int tx, int tiles) {
    constexpr int HC = CPL / 2, COLS = MtCols<CPL>::all, HALO = MtCols<CPL>::pre_halo;
    __shared__ __align__(16) T rows[MT_ROWS * COLS], rs[(MT_ROWS - MT_PRE_HALO + 2) * COLS / 2], zero[COLS], tab[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nrow = blockDim.x >> 5;
    MtRow<T, CPL> r;
    r.lane = lane;
    // the window's row of b that this warp holds
    auto place = [&](int t, int& g, int& c0) {
        c0 = (t % tx) * MtCols<CPL>::pre - HALO + CPL * lane;
        g = (t / tx) * (nrow - MT_PRE_HALO) - 5 + warp;
    };
    auto fetch = [&](int t, T* v) {
        int g, c0;
        place(t, g, c0);
        const int gw = g < F.ny + 5 ? mg_dom(g, F.ny, p.per_y) : -1;
#pragma unroll
        for (int k = 0; k < CPL; ++k) v[k] = T(0);
        if (gw >= 0 && c0 < F.nx + HALO) mt_load<CPL>(v, F.b, F.pitch, F.nx, gw, c0, c0 >= 0 && c0 + CPL - 1 < F.nx, p.per_x);
    };
    T bn[CPL];
    fetch(blockIdx.x, bn);
    if (threadIdx.x < COLS) zero[threadIdx.x] = T(0);
    if (warp == COLS / 32) tab[lane] = lane < 16 ? F.diag[lane] : F.invd[lane - 16];
    if (!block_live(S, inner)) return;
    const T scale = F.scale, ms = F.ms;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        place(t, r.g, r.c0);
        const int g0 = r.g - warp + 5;  // first row kept
        // (rows past the last one kept plus its halo have nothing to do)
        r.live = (p.per_y || (r.g >= 0 && r.g < F.ny)) && r.g < F.ny + 5;
        unsigned code;
        mt_open(r, F, p, tab, rows, zero, code);
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            r.x[k] = T(0);
            r.b[k] = bn[k];
        }
        if (t + (int)gridDim.x < tiles) fetch(t + gridDim.x, bn);
        if (r.live) r.template half<true>(0, scale);
        __syncthreads();
        auto in = [&](int k) { return r.live && warp >= k && warp < nrow - k; };
        if (in(1)) r.template half<false>(1, scale);
        __syncthreads();
        if (in(2)) r.template half<false>(0, scale);
        __syncthreads();
        if (in(3)) r.template half<false>(1, scale);
        __syncthreads();
        if (in(4)) {
            // x of the rows and columns kept
            const bool keep = in(5) && lane >= HALO / CPL && lane < 32 - HALO / CPL && r.g < F.ny;
            if (keep && r.c0 + CPL - 1 < F.nx) {
                mc_st<CPL>(F.r + (size_t)r.g * F.pitch + r.c0, r.x);
            } else if (keep) {
#pragma unroll
                for (int k = 0; k < CPL; ++k)
                    if (r.c0 + k < F.nx) F.r[(size_t)r.g * F.pitch + r.c0 + k] = r.x[k];
            }
            // residual, and the restriction's row sums under the lane's coarse
            // columns
            const T w = r.west(), e = r.east();
            T s[2][HC], m[2][HC], q[CPL];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int o = ((c + r.g + 1) & 1) * (COLS / 2);
                mc_ld<HC>(s[c], r.south + o);
                mc_ld<HC>(m[c], r.north + o);
            }
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                T ax = tab[code >> (4 * k) & 15u] * r.x[k];
                ax = mg_fma(ms, k == 0 ? w : r.x[(k + CPL - 1) % CPL], ax);
                ax = mg_fma(ms, k == CPL - 1 ? e : r.x[(k + 1) % CPL], ax);
                ax = mg_fma(ms, s[k & 1][k / 2], ax);
                ax = mg_fma(ms, m[k & 1][k / 2], ax);
                q[k] = r.b[k] - ax;
            }
            const T qw = __shfl_up_sync(0xffffffffu, q[CPL - 1], 1), qe = __shfl_down_sync(0xffffffffu, q[0], 1);
            T v[HC];
#pragma unroll
            for (int i = 0; i < HC; ++i) {
                // beside a wall the outer weight is 0 and the inner one the wall's
                const bool lo = !p.per_x && r.c0 + 2 * i == 0, hi = !p.per_x && r.c0 + 2 * i + 1 == F.nx - 1;
                T t2 = lo ? T(0) : mg_quarter(i == 0 ? qw : q[(2 * i + CPL - 1) % CPL]);
                t2 = mg_fma(lo && p.bc[0] == 0 ? T(1) : T(0.75), q[2 * i], t2);
                t2 = mg_fma(hi && p.bc[2] == 0 ? T(1) : T(0.75), q[2 * i + 1], t2);
                v[i] = mg_fma(hi ? T(0) : T(0.25), i == HC - 1 ? qe : q[(2 * i + 2) % CPL], t2);
            }
            mc_st<HC>(rs + (warp - 4) * (COLS / 2) + lane * HC, v);
        }
        __syncthreads();
        const int J = (g0 >> 1) + warp, nc = F.nx / 2, mc = F.ny / 2, I = (r.c0 >> 1);
        if (warp < (nrow - MT_PRE_HALO) / 2 && J < mc && lane >= HALO / CPL && lane < 32 - HALO / CPL && I < nc) {
            T wy[4], acc[HC];
#pragma unroll
            for (int i = 0; i < HC; ++i) acc[i] = T(0);
            mc_rweights<T>(J, mc, p.per_y, p.bc[1], p.bc[3], wy);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int g = 2 * J - 1 + a;
                if (!p.per_y && (g < 0 || g >= F.ny)) continue;
                T v[HC];
                mc_ld<HC>(v, rs + (2 * warp + a) * (COLS / 2) + lane * HC);
#pragma unroll
                for (int i = 0; i < HC; ++i) acc[i] = a == 0 ? mg_quarter(v[i]) : mg_fma(wy[a], v[i], acc[i]);
            }
            T* o = cb + (size_t)J * cpitch + I;
#pragma unroll
            for (int i = 0; i < HC; ++i)
                if (I + i < nc) o[i] = mg_quarter(acc[i]);
        }
    }
}

// A sum of FP32 terms in three words, each holding what the rounding of the one above
// left out: 72 bits, more than FP64's 53 (two words would hold 48), of FP32's range,
// as K1's p.q.  In FP64 a window's terms are 32 warp instructions of 64 cycles on four
// sub-partitions and the warps' totals 40 more: a 1024^2 mixed step 0.817 ms, this way
// 0.808 (0.813 with the warps' totals alone in FP64).
struct Sum72 {
    float h = 0.f, m = 0.f, l = 0.f;
    // s + v rounded, e what that left out
    __device__ __forceinline__ static float two_sum(float s, float v, float& e) {
        const float t = s + v, d = t - s;
        e = (s - (t - d)) + (v - d);
        return t;
    }
    __device__ __forceinline__ void add(float v) {
        float e, f;
        h = two_sum(h, v, e);
        m = two_sum(m, e, f);
        l = l + f;
    }
    // the warp's total, in every lane
    __device__ __forceinline__ double warp_total() {
#pragma unroll
        for (int k = 16; k >= 1; k >>= 1) {
            const float oh = __shfl_xor_sync(0xffffffffu, h, k), om = __shfl_xor_sync(0xffffffffu, m, k);
            const float ol = __shfl_xor_sync(0xffffffffu, l, k);
            float f;
            add(oh);
            m = two_sum(m, om, f);
            l = (l + ol) + f;
        }
        return (double)h + ((double)m + (double)l);
    }
};

// x = x_pre + P x_coarse, (black, red) x 2, x written; on the finest FP32 level
// also r.z and z's periodic ghosts (RzEpi)
template <typename T, int CPL>
__global__ void __launch_bounds__(MT_THREADS, 1) k_mg_post_rows(const T* cx, int cpitch, const __grid_constant__ MgLev<T> F,
                                                                MgBc p, SolverState* S, int inner, int tx, int tiles,
                                                                RzEpi E) {
    // hs: horizontal sums of the coarse rows under the window, row J at (J - J0) rows
    constexpr int HC = CPL / 2, COLS = MtCols<CPL>::all, HALO = MtCols<CPL>::post_halo;
    extern __shared__ __align__(16) unsigned char mt_smem[];
    T* const rows = reinterpret_cast<T*>(mt_smem);
    T* const hs = rows + MT_ROWS * COLS;
    __shared__ __align__(16) T zero[COLS], tab[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nrow = blockDim.x >> 5;
    MtRow<T, CPL> r;
    r.lane = lane;
    auto place = [&](int t, int& g, int& c0) {
        c0 = (t % tx) * MtCols<CPL>::post - HALO + CPL * lane;
        g = (t / tx) * (nrow - MT_POST_HALO) - 4 + warp;
    };
    auto fetch = [&](int t, T* bv, T* xv) {
        int g, c0;
        place(t, g, c0);
        const int gw = g < F.ny + 4 ? mg_dom(g, F.ny, p.per_y) : -1;
#pragma unroll
        for (int k = 0; k < CPL; ++k) bv[k] = xv[k] = T(0);
        if (gw >= 0 && c0 < F.nx + HALO) {
            const bool inside = c0 >= 0 && c0 + CPL - 1 < F.nx;
            mt_load<CPL>(bv, F.b, F.pitch, F.nx, gw, c0, inside, p.per_x);
            mt_load<CPL>(xv, F.r, F.pitch, F.nx, gw, c0, inside, p.per_x);
        }
    };
    T bn[CPL], xn[CPL];
    fetch(blockIdx.x, bn, xn);
    if (threadIdx.x < COLS) zero[threadIdx.x] = T(0);
    if (warp == COLS / 32) tab[lane] = lane < 16 ? F.diag[lane] : F.invd[lane - 16];
    if (!block_live(S, inner)) return;
    const T scale = F.scale;
    const int nc = F.nx / 2, mc = F.ny / 2;
    Sum72 rz;  // the lane's share of r.z
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        place(t, r.g, r.c0);
        r.live = (p.per_y || (r.g >= 0 && r.g < F.ny)) && r.g < F.ny + 4;
        unsigned code;
        mt_open(r, F, p, tab, rows, zero, code);
        const int J0 = ((r.g - warp) >> 1) - 1;  // coarse row below the window's first
        if (warp < nrow / 2 + 2) {
            const int Jw = J0 + warp < mc + 3 ? mg_dom(J0 + warp, mc, p.per_y) : -1;
            if (Jw >= 0) {
                const T* c = cx + (size_t)Jw * cpitch;
                const int I = r.c0 >> 1;
                auto at = [&](int i) {
                    i = i < nc + 4 ? mg_dom(i, nc, p.per_x) : -1;
                    return i >= 0 ? c[i] : T(0);
                };
                T m[HC];
                if (I >= 0 && I + HC - 1 < nc) {
                    mc_ld<HC>(m, c + I);
                } else {
#pragma unroll
                    for (int i = 0; i < HC; ++i) m[i] = at(I + i);
                }
                T w = __shfl_up_sync(0xffffffffu, m[HC - 1], 1), e = __shfl_down_sync(0xffffffffu, m[0], 1);
                if (lane == 0) w = at(I - 1);
                if (lane == 31) e = at(I + HC);
                // beside a SOLID wall the parent's weight is 1; beyond it the
                // neighbour is zero
                T h[CPL];
#pragma unroll
                for (int i = 0; i < HC; ++i) {
                    const T wl = (!p.per_x && I + i == 0 && p.bc[0] == 0) ? T(1) : T(0.75);
                    const T wr = (!p.per_x && I + i == nc - 1 && p.bc[2] == 0) ? T(1) : T(0.75);
                    h[2 * i] = mg_fma(T(0.25), i == 0 ? w : m[(i + HC - 1) % HC], wl * m[i]);
                    h[2 * i + 1] = mg_fma(T(0.25), i == HC - 1 ? e : m[(i + 1) % HC], wr * m[i]);
                }
                mc_st<CPL>(hs + warp * COLS + CPL * lane, h);
            }
        }
        __syncthreads();
        if (r.live) {
            const int J = r.g >> 1, NJ = J + ((r.g & 1) ? 1 : -1);
            const bool nin = p.per_y || (NJ >= 0 && NJ < mc);
            const T wyJ = (!nin && p.bc[NJ < 0 ? 1 : 3] == 0) ? T(1) : T(0.75);
            T h[CPL], n[CPL];
            mc_ld<CPL>(h, hs + (J - J0) * COLS + CPL * lane);
            if (nin) mc_ld<CPL>(n, hs + (NJ - J0) * COLS + CPL * lane);
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                T v = wyJ * h[k];
                if (nin) v = mg_fma(T(0.25), n[k], v);
                const bool cell = p.per_x || (r.c0 + k >= 0 && r.c0 + k < F.nx);
                r.x[k] = cell ? xn[k] + v : T(0);
                r.b[k] = bn[k];
            }
            r.store(0);
        }
        if (t + (int)gridDim.x < tiles) fetch(t + gridDim.x, bn, xn);
        __syncthreads();
        auto in = [&](int k) { return r.live && warp >= k && warp < nrow - k; };
        if (in(1)) r.template half<false>(1, scale);
        __syncthreads();
        if (in(2)) r.template half<false>(0, scale);
        __syncthreads();
        if (in(3)) r.template half<false>(1, scale);
        __syncthreads();
        if (in(4)) {
            r.template half<false>(0, scale);
            if (lane >= HALO / CPL && lane < 32 - HALO / CPL && r.g < F.ny) {
                T* row = F.x + (size_t)r.g * F.pitch;
                if (r.c0 + CPL - 1 < F.nx) {
                    mc_st<CPL>(row + r.c0, r.x);
                } else {
#pragma unroll
                    for (int k = 0; k < CPL; ++k)
                        if (r.c0 + k < F.nx) row[r.c0 + k] = r.x[k];
                }
                if (sizeof(T) == 4 && E.on) {
#pragma unroll
                    for (int k = 0; k < CPL; ++k) {
                        const int gi = r.c0 + k, gj = r.g;
                        if (gi >= F.nx) continue;
                        // ghost copies along periodic axes (the finest level's x has a ghost ring)
                        if (p.per_x) {
                            if (gi == 0) row[F.nx] = r.x[k];
                            if (gi == F.nx - 1) row[-1] = r.x[k];
                        }
                        if (p.per_y) {
                            if (gj == 0) F.x[(ptrdiff_t)F.ny * F.pitch + gi] = r.x[k];
                            if (gj == F.ny - 1) F.x[-(ptrdiff_t)F.pitch + gi] = r.x[k];
                        }
                    }
                }
            }
        }
        if (sizeof(T) == 4 && E.on) {
            // r.z in units of two cells eight rows apart, one fused operation each (the
            // solver's fixed FP32 order; windows of MT_RZ_ROWS hold whole units)
            constexpr int lo = MT_POST_HALO / 2;
            const bool own = lane >= HALO / CPL && lane < 32 - HALO / CPL && r.g < F.ny;
            if (warp >= lo && warp < lo + 8) {
                T v[CPL];
#pragma unroll
                for (int k = 0; k < CPL; ++k) v[k] = own && r.c0 + k < F.nx ? mg_fma(r.b[k], r.x[k], T(0)) : T(0);
                mc_st<CPL>(hs + (warp - lo) * COLS + CPL * lane, v);
            }
            __syncthreads();
            if (warp >= lo + 8 && warp < lo + 16) {
                T v[CPL];
                mc_ld<CPL>(v, hs + (warp - lo - 8) * COLS + CPL * lane);
#pragma unroll
                for (int k = 0; k < CPL; ++k) {
                    if (own && r.c0 + k < F.nx) v[k] = mg_fma(r.b[k], r.x[k], v[k]);
                    rz.add((float)v[k]);
                }
            }
            __syncthreads();
        }
    }
    if (sizeof(T) == 4 && E.on) {
        double v[1] = {0.0};
        // (the other warps hold nothing)
        if (warp >= MT_POST_HALO / 2 + 8 && warp < MT_POST_HALO / 2 + 16) v[0] = rz.warp_total();
        const double den = S->refreshed ? S->rho_prev : S->rho_in;
        if (grid_totals<1, MT_ROWS>(v, E.part, nullptr, &S->ticket[7]) && threadIdx.x == 0) rz_scalars(S, v[0], den);
    }
}

template <typename T, int CPL>
constexpr size_t MT_POST_SMEM = sizeof(T) * (MT_ROWS + MT_ROWS / 2 + 2) * MtCols<CPL>::all;

// Windows of a level: their count, the count per row of them, their rows (even) and
// columns per lane, chosen so that the blocks (one to an SM) finish first.  A window
// costs its rows times its columns and as much again in barriers and latency as `more`
// rows; the choice is flat in it (a 1024^2 mixed step is 0.797 to 0.808 ms and a 4096^2
// one 2.527 to 2.533 with 8, 16, 24 or 40, an FP64 one the same with 2, 4 or 8).  FP64 may take two columns to a lane: a small level then has narrower
// and taller windows, less of them halo (256^2 10.1 -> 7.9 us each way, 128^2 7.9 ->
// 6.1, 192x160 9.1 -> 6.7; 512^2 keeps four, 18 and 17 us).
struct MtGrid {
    int tx, tiles, rows, cpl;
};
template <typename T>
static MtGrid mt_grid(int nx, int ny, int sms, bool pre, int fixed_rows = 0) {
    const int halo = pre ? MT_PRE_HALO : MT_POST_HALO, more = sizeof(T) == 4 ? 16 : 4;
    MtGrid best{};
    long long cost = -1;
    for (int cpl : {4, 2}) {
        if (cpl == 2 && sizeof(T) == 4) continue;
        const int w = cpl == 4 ? (pre ? MtCols<4>::pre : MtCols<4>::post) : (pre ? MtCols<2>::pre : MtCols<2>::post);
        const int tx = (nx + w - 1) / w;
        for (int rows = MT_ROWS; rows >= halo + 2; rows -= 2) {
            if (fixed_rows > 0 && rows != fixed_rows) continue;
            const int tiles = tx * ((ny + rows - halo - 1) / (rows - halo));
            const long long c = (long long)((tiles + sms - 1) / sms) * (rows + more) * cpl;
            if (cost < 0 || c < cost) {
                cost = c;
                best = MtGrid{tx, tiles, rows, cpl};
            }
        }
    }
    return best;
}
