// The coarse half of the multigrid V-cycle in one launch: a thread-block
// cluster keeps every level from the first small one down to the coarsest in
// distributed shared memory (included by cf_mg.cu, whose per-cell arithmetic
// and operation order it repeats, so each value is the one the launch-per-level
// kernels form).
//
// Why: a small level is latency.  As launches of shared-memory tiles, each level
// below 256^2 cost 6.5-7 us per direction in FP32 (9-12 us in FP64) and a one-CTA
// solver of the last ones 34 us (45-65 us): 74 us of an FP32 V-cycle and 128 us of
// an FP64 one from 256^2 and 128^2.  Inside a cluster the levels meet at a hardware
// barrier (0.2 us) and read each other's rows directly: 20 us (FP32 from 128^2; 29 us
// between the launches of a 4096^2 cycle, whose traffic leaves the caches cold) and
// 33 us (FP64 from 64^2), 10 and 17 us when only the levels from 32^2 and 16^2 are
// there.
//
// Levels [0, ns) are distributed: a CTA owns a band of rows (twice as many on
// each finer level).  Within a level no CTA waits for another: MC_H halo rows
// are recomputed, one row fewer per half sweep (5, 4, 3, 2 rows on the way
// down, 3, 2, 1, 0 on the way up), as the tile kernels do; between levels the
// halo rows are read from their owners' shared memory.  A warp holds one row
// (band or halo) in registers, CPL consecutive columns to a lane: the west and
// east neighbours are its own or come by shuffle, the rows above and below
// through shared memory, where a row keeps its red and its black cells apart.
// (A form that kept x and b in shared memory and read five neighbours there
// spent 1650 cycles on a 256-wide half sweep, all of it shared-memory
// wavefronts.)  Levels [ns, nlev) are solved by CTA 0 alone, one cell pair per
// thread, with barriers of just the warps that hold cells; a coarsest level of
// at most 32 pairs stays in one warp's registers.
#pragma once

constexpr int MC_LEVELS = 8;
constexpr int MC_H = 5;
constexpr int MC_THREADS = 1024;
constexpr long long MC_COARSEST = 1024;  // cells of the coarsest level at most
constexpr int MC_WARPS = MC_THREADS / 32;

// Largest first level, its most columns (32 lanes of CPL), and the level size
// CTA 0 takes alone.  A cluster is 16 of the SMs and recomputes its halo rows, so a
// level goes there only once its launches (cf_mgt.cuh) are latency too.  FP32:
// 128^2 (a 1024^2 step 0.797 ms, with 256^2 in the cluster 0.806, from 64^2 on 0.807;
// 4096^2 2.535, 2.549, 2.529).  FP64, where an SM executes two operations per cycle:
// 64^2 (a 192x160 step 0.617 ms, without 48x40 0.628; 512^2 adjoint 7.90 + 12.35, 7.95
// + 12.40; with 96x80 and 128^2 in it, before these levels had narrow windows, 0.737
// against 0.682 and 8.58 + 13.15 against 8.34 + 12.88); alone up to 16^2 for
// the same reason.
template <typename T>
struct McMax {
    static constexpr int first = sizeof(T) == 4 ? 16384 : 4096;
    static constexpr int columns = sizeof(T) == 4 ? 256 : 128;
    static constexpr int alone = sizeof(T) == 4 ? 1024 : 256;
    static_assert(alone <= 2 * MC_THREADS, "a thread of CTA 0 holds one cell pair");
};

template <typename T>
struct MgCoarse {
    int nlev, ns;
    int nx[MC_LEVELS], ny[MC_LEVELS];
    int cpl[MC_LEVELS];             // distributed: columns per lane (2, 4, 8), negative where nx is less than 32 of them
    int sp[MC_LEVELS];              // row pitch in shared memory (elements)
    int xo[MC_LEVELS], bo[MC_LEVELS];  // offsets of x and b (elements)
    unsigned inv[MC_LEVELS];        // levels of CTA 0: ceil(2^20 / pairs per row)
    int cxo;                        // the band of level ns's x, on every CTA
    int tmp;                        // row sums; CTA 0's residuals
    int zero;                       // a row of zeros (beyond a wall)
    T scale[MC_LEVELS], ms[MC_LEVELS];
    // diagonal and its reciprocal by the number of SOLID sides; which sides are
    T dv[MC_LEVELS][10];
    int solid;
    const T* gb;                    // level 0: right-hand side in, x out
    T* gx;
    int gpitch;
};

__device__ __forceinline__ void mc_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void mc_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned mc_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned mc_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// this CTA's shared-memory address seen in another CTA of the cluster, and a
// store there
template <typename T>
__device__ __forceinline__ unsigned mc_map(const T* p, unsigned rank) {
    unsigned q;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(q)
                 : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return q;
}
__device__ __forceinline__ void mc_put(const float* p, unsigned rank, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mc_map(p, rank)), "f"(v) : "memory");
}
__device__ __forceinline__ void mc_put(const double* p, unsigned rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(mc_map(p, rank)), "d"(v) : "memory");
}
// a barrier of the first n threads (n a multiple of 32), one id per level
__device__ __forceinline__ void mc_bar(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// columns of padding before column 0 of a row of CTA 0's levels (16 bytes)
template <typename T>
struct McPad {
    static constexpr int value = 16 / (int)sizeof(T);
};

// N values between shared memory and registers, in vectors of up to 16 bytes
// (addresses are multiples of the vector size)
template <int N>
__device__ __forceinline__ void mc_ld(float* v, const float* p) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 4) {
            const float4 q = *reinterpret_cast<const float4*>(p + k);
            v[k] = q.x;
            v[k + 1] = q.y;
            v[k + 2] = q.z;
            v[k + 3] = q.w;
        }
    } else if constexpr (N == 2) {
        const float2 q = *reinterpret_cast<const float2*>(p);
        v[0] = q.x;
        v[1] = q.y;
    } else {
        v[0] = p[0];
    }
}
template <int N>
__device__ __forceinline__ void mc_ld(double* v, const double* p) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 2) {
            const double2 q = *reinterpret_cast<const double2*>(p + k);
            v[k] = q.x;
            v[k + 1] = q.y;
        }
    } else {
        v[0] = p[0];
    }
}
template <int N>
__device__ __forceinline__ void mc_st(float* p, const float* v) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 4) *reinterpret_cast<float4*>(p + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else if constexpr (N == 2) {
        *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    } else {
        p[0] = v[0];
    }
}
template <int N>
__device__ __forceinline__ void mc_st(double* p, const double* v) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 2) *reinterpret_cast<double2*>(p + k) = make_double2(v[k], v[k + 1]);
    } else {
        p[0] = v[0];
    }
}

// one row of n16 16-byte pieces from another CTA's shared memory (src: its
// address in the cluster's window) to this CTA's, by one warp
template <typename T>
__device__ __forceinline__ void mc_row(T* dst, unsigned src, int n16) {
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll 4
    for (int i = threadIdx.x & 31; i < n16; i += 32) {
        uint4 v;
        asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(src + 16u * i)
                     : "memory");
        d[i] = v;
    }
}

// What the distributed levels share: the band's rows per level (start[c] on
// level ns, doubled on each finer level) and the tables.
template <typename T>
struct McCta {
    T* sm;
    const T* tab;         // per level: diag[16], 1 / diag[16]
    const int* start;     // band starts on level ns, C + 1 entries
    const short* own;     // owner of each row of level ns
    int rank, ns;
};

// The halo rows [j0 - ext, j0) and [j1, j1 + ext) of an array of level l (row
// g at off + (g - j0 + MC_H) sp) from the CTAs that own them; warps take rows
// from warp w0 on.
template <typename T>
__device__ __forceinline__ void mc_pull(const MgCoarse<T>& P, const MgBc& p, const McCta<T>& K, int l, int off, int ext,
                                        int w0) {
    const int ny = P.ny[l], sp = P.sp[l], shift = K.ns - l;
    const int j0 = K.start[K.rank] << shift, j1 = K.start[K.rank + 1] << shift;
    const int k = (int)(threadIdx.x >> 5) - w0;
    if (j0 == j1 || k < 0 || k >= 2 * ext) return;
    const int g = k < ext ? j0 - ext + k : j1 + (k - ext);
    int gw = g;
    if (g < 0 || g >= ny) {
        if (!p.per_y) return;
        gw = g < 0 ? g + ny : g - ny;
    }
    const int o = K.own[gw >> shift];
    const unsigned src = mc_map(K.sm + off + (gw - (K.start[o] << shift) + MC_H) * sp, (unsigned)o);
    mc_row(K.sm + off + (g - j0 + MC_H) * sp, src, sp * (int)sizeof(T) / 16);
}

// restriction weights of coarse index I along one axis (quarters as in
// mg_pwq): fine cells 2I - 1 .. 2I + 2
template <typename T>
__device__ __forceinline__ void mc_rweights(int I, int nc, int per, int bclo, int bchi, T* w) {
    const bool lo = I == 0 && !per, hi = I == nc - 1 && !per;
    w[0] = lo ? T(0) : T(0.25);
    w[1] = (lo && bclo == 0) ? T(1) : T(0.75);
    w[2] = (hi && bchi == 0) ? T(1) : T(0.75);
    w[3] = hi ? T(0) : T(0.25);
}

// A warp's row of a distributed level: lane l holds columns CPL l .. CPL l +
// CPL - 1 (columns past the grid hold zero), row g in the band's coordinates
// (wrapped rows keep their unwrapped number; ny is even, so the parity holds).
// In shared memory a row is its red cells (gi + g even) and then its black
// ones, CPL / 2 of each per lane.  FULL: the grid fills the 32 lanes.  What
// bounds a half sweep is instruction issue (26 warps on one SM at 256 columns),
// so boundary logic is kept out of it: the rows beyond a wall read as a row of
// zeros, and only the lane at the row's end looks at the wall.
template <typename T, int CPL, bool FULL>
struct McRow {
    static constexpr int HC = CPL / 2;
    int nx, g, col0, sp, lane, per_x;
    bool live;                    // the row exists
    T* row;                       // this row in shared memory, at the lane's cells
    const T *south, *north;       // the rows below and above, likewise
    T idm, idw, ide;              // 1 / diagonal: inside, first column, last column
    T x[CPL], b[CPL];

    __device__ __forceinline__ T west() const {  // of the lane's first column
        if (FULL) {
            const T v = __shfl_sync(0xffffffffu, x[CPL - 1], (lane + 31) & 31);
            return (lane == 0 && !per_x) ? T(0) : v;
        }
        T v = __shfl_up_sync(0xffffffffu, x[CPL - 1], 1);
        if (lane == 0) v = T(0);
        if (per_x) {
            T e = T(0);
#pragma unroll
            for (int k = 1; k < CPL; k += 2)
                if ((nx - 1) % CPL == k) e = x[k];
            e = __shfl_sync(0xffffffffu, e, (nx - 1) / CPL);
            if (lane == 0) v = e;
        }
        return v;
    }
    __device__ __forceinline__ T east() const {  // of the lane's last column in the grid
        if (FULL) {
            const T v = __shfl_sync(0xffffffffu, x[0], (lane + 1) & 31);
            return (lane == 31 && !per_x) ? T(0) : v;
        }
        T v = __shfl_down_sync(0xffffffffu, x[0], 1);
        if (lane == 31) v = T(0);
        if (per_x) {
            const T f = __shfl_sync(0xffffffffu, x[0], 0);
            if (col0 + CPL >= nx) v = f;
        }
        return v;
    }
    // column col0 + k is the row's last one
    __device__ __forceinline__ bool end(int k) const {
        return FULL ? (k == CPL - 1 && lane == 31) : col0 + k == nx - 1;
    }
    // column k's neighbour to the east; e: the lane's
    __device__ __forceinline__ T right(int k, T e) const {
        if (k == CPL - 1) return e;
        return (!FULL && per_x && end(k)) ? e : x[(k + 1) % CPL];
    }
    __device__ __forceinline__ T mask(int k, T v) const { return (FULL || col0 + k < nx) ? v : T(0); }
    // the cells of one colour to shared memory
    __device__ __forceinline__ void store(int color) const {
        T v[HC];
        const int sel = (g + color) & 1;
#pragma unroll
        for (int i = 0; i < HC; ++i) v[i] = sel ? x[2 * i + 1] : x[2 * i];
        mc_st<HC>(row + color * (sp / 2), v);
    }
    // half sweep of one colour; the rows above and below hold the other one
    // (FIRST: from x = 0)
    template <bool FIRST>
    __device__ __forceinline__ void half(int color, T scale) {
        T s[HC], n[HC], v[HC];
        if (!FIRST) {
            mc_ld<HC>(s, south + (1 - color) * (sp / 2));
            mc_ld<HC>(n, north + (1 - color) * (sp / 2));
        }
        if (((g + color) & 1) == 0) {  // the cells over even columns
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
                v[i] = x[2 * i] = mask(2 * i, t * ((i == 0 && lane == 0) ? idw : idm));
            }
        } else {
            const T e = FIRST ? T(0) : east();
#pragma unroll
            for (int i = 0; i < HC; ++i) {
                const int k = 2 * i + 1;
                T t = b[k];
                if (!FIRST) {
                    t = x[k - 1] + right(k, e);
                    t = t + s[i];
                    t = t + n[i];
                    t = mg_fma(scale, t, b[k]);
                }
                v[i] = x[k] = mask(k, t * ((!FULL || k == CPL - 1) && end(k) ? ide : idm));
            }
        }
        mc_st<HC>(row + color * (sp / 2), v);
    }
};

// a warp's row of level l: row warp of the band with its halo
template <typename T, int CPL, bool FULL>
__device__ __forceinline__ void mc_open(const MgCoarse<T>& P, const MgBc& p, const McCta<T>& K, int l,
                                        McRow<T, CPL, FULL>& r) {
    const int shift = K.ns - l, j0 = K.start[K.rank] << shift, j1 = K.start[K.rank + 1] << shift;
    const int warp = threadIdx.x >> 5;
    r.lane = threadIdx.x & 31;
    r.nx = P.nx[l];
    r.sp = P.sp[l];
    r.per_x = p.per_x;
    r.g = j0 - MC_H + warp;
    r.col0 = CPL * r.lane;
    const int ny = P.ny[l];
    r.live = j0 < j1 && r.g < j1 + MC_H && (p.per_y || (r.g >= 0 && r.g < ny));
    const bool wall_s = !p.per_y && r.g == 0, wall_n = !p.per_y && r.g == ny - 1;
    const T* zero = K.sm + P.zero + r.lane * (CPL / 2);
    r.row = K.sm + P.xo[l] + warp * r.sp + r.lane * (CPL / 2);
    r.south = wall_s ? zero : r.row - r.sp;
    r.north = wall_n ? zero : r.row + r.sp;
    const int rb = (wall_s ? 4 : 0) | (wall_n ? 8 : 0);
    const T* invd = K.tab + l * 32 + 16;
    r.idm = invd[rb];
    r.idw = invd[rb | (p.per_x ? 0 : 1)];
    r.ide = invd[rb | (p.per_x ? 0 : 2)];
#pragma unroll
    for (int k = 0; k < CPL; ++k) r.x[k] = T(0);
    if (r.live) mc_ld<CPL>(r.b, K.sm + P.bo[l] + warp * r.sp + r.col0);
}

// Down one distributed level: x = 4 half sweeps from 0 (kept in shared memory
// for the way up), r = b - A x, and the restriction of the band's coarse rows
// to the next level's b.
template <typename T, int CPL, bool FULL>
__device__ __forceinline__ void mc_down(const MgCoarse<T>& P, const MgBc& p, const McCta<T>& K, int l) {
    constexpr int HC = CPL / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int shift = K.ns - l, n = (K.start[K.rank + 1] - K.start[K.rank]) << shift;
    const int J0 = K.start[K.rank] << shift >> 1, nc = P.nx[l + 1], mc = P.ny[l + 1];
    McRow<T, CPL, FULL> r;
    mc_open(P, p, K, l, r);
    const T scale = P.scale[l], ms = P.ms[l];
    // rows of the band grown by ext
    const int dist = !r.live ? 1 << 20 : (warp < MC_H ? MC_H - warp : warp - (MC_H + n) + 1);
    if (dist <= 5) r.template half<true>(0, scale);
    __syncthreads();
    if (dist <= 4) r.template half<false>(1, scale);
    __syncthreads();
    if (dist <= 3) r.template half<false>(0, scale);
    __syncthreads();
    if (dist <= 2) r.template half<false>(1, scale);
    __syncthreads();
    // residual of the band and a row to each side, and the restriction's row
    // sums under the lane's coarse columns
    T* rs = K.sm + P.tmp;  // row warp at warp * 32 HC
    if (dist <= 1) {
        const T* diag = K.tab + l * 32;
        const int rb = p.per_y ? 0 : (r.g == 0 ? 4 : 0) | (r.g == P.ny[l] - 1 ? 8 : 0);
        const T dm = diag[rb], dw = diag[rb | (p.per_x ? 0 : 1)], de = diag[rb | (p.per_x ? 0 : 2)];
        const T w = r.west(), e = r.east();
        T s[2][HC], m[2][HC];  // rows below and above: the cells over even and odd columns
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int o = ((c + r.g + 1) & 1) * (r.sp / 2);  // column parity c of row g +- 1 has this colour
            mc_ld<HC>(s[c], r.south + o);
            mc_ld<HC>(m[c], r.north + o);
        }
        T q[CPL];
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            T d = dm;
            if (k == 0 && lane == 0) d = dw;
            if ((!FULL || k == CPL - 1) && r.end(k)) d = de;
            T ax = d * r.x[k];
            ax = mg_fma(ms, k == 0 ? w : r.x[(k + CPL - 1) % CPL], ax);
            ax = mg_fma(ms, r.right(k, e), ax);
            ax = mg_fma(ms, s[k & 1][k / 2], ax);
            ax = mg_fma(ms, m[k & 1][k / 2], ax);
            q[k] = r.mask(k, r.b[k] - ax);
        }
#pragma unroll
        for (int k = 0; k < CPL; ++k) r.x[k] = q[k];  // (its west and east by the same exchange)
        const T qw = r.west(), qe = r.east();
        T v[HC];
#pragma unroll
        for (int i = 0; i < HC; ++i) {
            // weights 1/4, 3/4, 3/4, 1/4; beside a wall the outer one is 0 and
            // the inner one the wall's
            const bool lo = i == 0 && lane == 0 && !p.per_x;
            const bool hi = (!FULL || i == HC - 1) && !p.per_x && r.end(2 * i + 1);
            T t = lo ? T(0) : mg_quarter(i == 0 ? qw : q[(2 * i + CPL - 1) % CPL]);
            t = mg_fma(lo && p.bc[0] == 0 ? T(1) : T(0.75), q[2 * i], t);
            t = mg_fma(hi && p.bc[2] == 0 ? T(1) : T(0.75), q[2 * i + 1], t);
            v[i] = mg_fma(hi ? T(0) : T(0.25), r.right(2 * i + 1, qe), t);
        }
        mc_st<HC>(rs + warp * 32 * HC + lane * HC, v);
    }
    __syncthreads();
    if (warp < n / 2) {
        const int J = J0 + warp;
        T wy[4], acc[HC];
        mc_rweights<T>(J, mc, p.per_y, p.bc[1], p.bc[3], wy);
#pragma unroll
        for (int i = 0; i < HC; ++i) acc[i] = T(0);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int g = 2 * J - 1 + a;
            if (!p.per_y && (g < 0 || g >= P.ny[l])) continue;
            T v[HC];
            mc_ld<HC>(v, rs + (2 * warp - 1 + a + MC_H) * 32 * HC + lane * HC);
#pragma unroll
            for (int i = 0; i < HC; ++i) acc[i] = a == 0 ? mg_quarter(v[i]) : mg_fma(wy[a], v[i], acc[i]);
        }
#pragma unroll
        for (int i = 0; i < HC; ++i) acc[i] = mg_quarter(acc[i]);
        if (l + 1 < K.ns) {
            mc_st<HC>(K.sm + P.bo[l + 1] + (warp + MC_H) * P.sp[l + 1] + lane * HC, acc);
        } else {
#pragma unroll
            for (int i = 0; i < HC; ++i)
                if (lane * HC + i < nc)
                    mc_put(K.sm + P.bo[K.ns] + J * P.sp[K.ns] + McPad<T>::value + lane * HC + i, 0u, acc[i]);
        }
    }
}

// Up one distributed level: x += P x_coarse on the band and four rows to each
// side, 4 half sweeps; the band's x to global memory (level 0), or over b's
// rows, in column order, for the next finer level.
template <typename T, int CPL, bool FULL>
__device__ __forceinline__ void mc_up(const MgCoarse<T>& P, const MgBc& p, const McCta<T>& K, int l) {
    constexpr int HC = CPL / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int shift = K.ns - l, n = (K.start[K.rank + 1] - K.start[K.rank]) << shift;
    const int J0 = K.start[K.rank] << shift >> 1, J1 = J0 + n / 2, nc = P.nx[l + 1], mc = P.ny[l + 1];
    McRow<T, CPL, FULL> r;
    mc_open(P, p, K, l, r);
    const T scale = P.scale[l];
    const int dist = !r.live ? 1 << 20 : (warp < MC_H ? MC_H - warp : warp - (MC_H + n) + 1);
    // the horizontal sums of coarse rows J0 - 3 .. J1 + 2, one warp each (row J
    // of the band: b's place on a distributed level, cxo for level ns)
    T* hs = K.sm + P.tmp;  // row J at (J - J0 + 3) * 32 CPL
    {
        const int J = J0 - 3 + warp, csp = P.sp[l + 1];
        if (J < J1 + 3 && n > 0 && (p.per_y || (J >= 0 && J < mc))) {
            const T* c = K.sm + (l + 1 < K.ns ? P.bo[l + 1] : P.cxo + McPad<T>::value) + (J - J0 + MC_H) * csp;
            T m[HC], h[CPL];
            mc_ld<HC>(m, c + lane * HC);
#pragma unroll
            for (int i = 0; i < HC; ++i) m[i] = (FULL || lane * HC + i < nc) ? m[i] : T(0);
            T w = __shfl_up_sync(0xffffffffu, m[HC - 1], 1), e = __shfl_down_sync(0xffffffffu, m[0], 1);
            if (lane == 0) w = p.per_x ? c[nc - 1] : T(0);
            const T f = p.per_x ? c[0] : T(0);  // east of the last coarse column
#pragma unroll
            for (int i = 0; i < HC; ++i) {
                const bool last = (!FULL || i == HC - 1) && r.end(2 * i + 1);
                const T wl = (i == 0 && lane == 0 && !p.per_x && p.bc[0] == 0) ? T(1) : T(0.75);
                const T wr = (last && !p.per_x && p.bc[2] == 0) ? T(1) : T(0.75);
                h[2 * i] = mg_fma(T(0.25), i == 0 ? w : m[(i + HC - 1) % HC], wl * m[i]);
                h[2 * i + 1] = mg_fma(T(0.25), last ? f : (i == HC - 1 ? e : m[(i + 1) % HC]), wr * m[i]);
            }
            mc_st<CPL>(hs + warp * 32 * CPL + lane * CPL, h);
        }
    }
    __syncthreads();
    if (dist <= 4) {
        T v[2][HC], h[CPL], k1[CPL];
#pragma unroll
        for (int c = 0; c < 2; ++c) mc_ld<HC>(v[c], r.row + ((c + r.g) & 1) * (r.sp / 2));  // the kept x, column parity c
        const int J = r.g >> 1, NJ = J + ((r.g & 1) ? 1 : -1);
        const bool nin = p.per_y || (NJ >= 0 && NJ < mc);
        const T wyJ = (!nin && p.bc[NJ < 0 ? 1 : 3] == 0) ? T(1) : T(0.75);
        mc_ld<CPL>(h, hs + (J - J0 + 3) * 32 * CPL + lane * CPL);
        if (nin) mc_ld<CPL>(k1, hs + (NJ - J0 + 3) * 32 * CPL + lane * CPL);
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            T t = wyJ * h[k];
            if (nin) t = mg_fma(T(0.25), k1[k], t);
            r.x[k] = r.mask(k, v[k & 1][k / 2] + t);
        }
        r.store(0);
    }
    __syncthreads();
    if (dist <= 3) r.template half<false>(1, scale);
    __syncthreads();
    if (dist <= 2) r.template half<false>(0, scale);
    __syncthreads();
    if (dist <= 1) r.template half<false>(1, scale);
    __syncthreads();
    if (dist <= 0) {
        r.template half<false>(0, scale);
        if (l == 0) {
            T* x = P.gx + (size_t)r.g * P.gpitch + r.col0;
            if (FULL || r.col0 + CPL <= r.nx) {
                mc_st<CPL>(x, r.x);
            } else {
#pragma unroll
                for (int k = 0; k < CPL; ++k)
                    if (r.col0 + k < r.nx) x[k] = r.x[k];
            }
        } else {
            mc_st<CPL>(K.sm + P.bo[l] + warp * r.sp + r.col0, r.x);
        }
    }
}

// one cell pair (red and black) of a level CTA 0 holds alone
template <typename T>
struct McPair {
    int c[2], w[2], e[2], s[2], n[2];  // offsets in x: the cell and its neighbours
    T id[2], d[2], b[2];
    bool in[2];
};

template <typename T>
__global__ void __launch_bounds__(MC_THREADS, 1) k_mg_coarse(const __grid_constant__ MgCoarse<T> P, MgBc p,
                                                              SolverState* S, int inner) {
    extern __shared__ __align__(16) unsigned char mc_smem[];
    T* sm = reinterpret_cast<T*>(mc_smem);
    __shared__ __align__(16) T tab[MC_LEVELS * 32];  // per level: diag[16], 1 / diag[16]
    __shared__ int start[MC_WARPS + 1];
    __shared__ short own[MC_COARSEST];
    __shared__ int live;
    constexpr int PAD = McPad<T>::value;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)mc_rank(), C = (int)mc_size();
    const int ns = P.ns, nlev = P.nlev, base = P.ny[ns];
    // level 0's right-hand side comes in and the solver status is fetched while
    // the rest is set up
    {
        const int n0 = ns > 0 ? (rank * base / C) << ns : 0, n1 = ns > 0 ? ((rank + 1) * base / C) << ns : P.ny[0];
        const int h = ns > 0 ? MC_H : 0, off = ns > 0 ? 0 : PAD, nx = P.nx[0];
        for (int g = n0 - h + warp; g < n1 + h && n0 < n1; g += MC_WARPS) {
            const int gw = mg_dom(g, P.ny[0], p.per_y);
            if (gw < 0) continue;
            const T* src = P.gb + (size_t)gw * P.gpitch;
            T* dst = sm + P.bo[0] + (g - n0 + h) * P.sp[0] + off;
            for (int i = lane * PAD; i < P.sp[0] - off; i += 32 * PAD) {
                if (i + PAD <= nx)
                    cpa16(dst + i, src + i);
                else
                    for (int k = 0; k < PAD; ++k) dst[i + k] = i + k < nx ? src[i + k] : T(0);
            }
        }
        cpa_commit();
    }
    int st = ST_RUNNING, ist = ST_RUNNING;
    if (tid == 0) {
        st = *(volatile const int*)&S->status;
        if (inner) ist = *(volatile const int*)&S->inner_status;
    }
    if (tid <= C) start[tid] = (tid * base) / C;
    if (tid < base) own[tid] = (short)(((tid + 1) * C - 1) / base);
    if (warp < nlev) {  // one level's tables, lane = entry
        const int sides = __popc(lane & 15 & P.solid);
        const T* v = P.dv[warp];
        const bool recip = lane & 16;
        T t = recip ? v[5] : v[0];
#pragma unroll
        for (int k = 1; k < 5; ++k)
            if (sides == k) t = recip ? v[5 + k] : v[k];
        tab[warp * 32 + lane] = t;
    }
    if (ns > 0)
        for (int k = tid; k < P.sp[0]; k += MC_THREADS) sm[P.zero + k] = T(0);
    // CTA 0's levels: x starts at zero, and so does the padding beyond a wall
    if (rank == 0)
        for (int l = ns; l < nlev; ++l)
            for (int k = P.xo[l] + PAD * tid; k < P.bo[l]; k += PAD * MC_THREADS)
                *reinterpret_cast<uint4*>(sm + k) = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) live = st == ST_RUNNING && ist == ST_RUNNING;
    cpa_wait<0>();
    __syncthreads();
    if (!live) return;  // the same answer in every CTA
    mc_arrive();
    const McCta<T> K{sm, tab, start, own, rank, ns};
    mc_wait();  // every CTA is up before another touches its memory
    // ---- down, distributed levels
    for (int l = 0; l < ns; ++l) {
        switch (P.cpl[l]) {  // negative: the grid does not fill the lanes
            case 2: mc_down<T, 2, true>(P, p, K, l); break;
            case 4: mc_down<T, 4, true>(P, p, K, l); break;
            case -2: mc_down<T, 2, false>(P, p, K, l); break;
            case -4: mc_down<T, 4, false>(P, p, K, l); break;
            case 8:
                if constexpr (sizeof(T) == 4) mc_down<T, 8, true>(P, p, K, l);
                break;
            default:
                if constexpr (sizeof(T) == 4) mc_down<T, 8, false>(P, p, K, l);
        }
        mc_arrive();
        mc_wait();
        // the next level's right-hand side with its halo, and (x is final until
        // the way up) x's halo for the post-smoothing; CTA 0 goes on to its own
        // levels first
        if (l + 1 < ns) {
            mc_pull(P, p, K, l + 1, P.bo[l + 1], MC_H, 0);
            mc_pull(P, p, K, l, P.xo[l], 4, 2 * MC_H);
            __syncthreads();
        }
    }
    // ---- the levels of CTA 0
    if (rank == 0) {
        auto pairs_of = [&](int l) { return ((P.nx[l] + 1) / 2) * P.ny[l]; };
        auto row_of = [&](int l) { return (int)((unsigned)tid * P.inv[l] >> 20); };  // tid / pairs per row
        auto make = [&](int l, McPair<T>& q) {
            const int nx = P.nx[l], ny = P.ny[l], sp = P.sp[l], hw = (nx + 1) / 2;
            const int gj = row_of(l), pr = tid - gj * hw;
            const T* b = sm + P.bo[l] + PAD;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int gi = 2 * pr + ((gj + k) & 1);
                q.in[k] = gj < ny && gi < nx;
                const int o = P.xo[l] + (gj + 1) * sp + PAD;  // column 0 of the row
                const bool w = gi == 0, e = gi == nx - 1, s = gj == 0, n = gj == ny - 1;
                q.c[k] = o + gi;
                q.w[k] = o + ((w && p.per_x) ? nx - 1 : gi - 1);
                q.e[k] = o + ((e && p.per_x) ? 0 : gi + 1);
                q.s[k] = o + gi + ((s && p.per_y) ? (ny - 1) * sp : -sp);
                q.n[k] = o + gi + ((n && p.per_y) ? -(ny - 1) * sp : sp);
                const int bits = (p.per_x ? 0 : (w ? 1 : 0) | (e ? 2 : 0)) | (p.per_y ? 0 : (s ? 4 : 0) | (n ? 8 : 0));
                q.id[k] = tab[l * 32 + 16 + bits];
                q.d[k] = tab[l * 32 + bits];
                q.b[k] = q.in[k] ? b[gj * sp + gi] : T(0);
            }
        };
        auto half = [&](const McPair<T>& q, int k, T scale, bool first) {
            if (!q.in[k]) return;
            T s;
            if (first) {
                s = T(0);
            } else {
                s = sm[q.w[k]] + sm[q.e[k]];
                s = s + sm[q.s[k]];
                s = s + sm[q.n[k]];
            }
            const T t = mg_fma(scale, s, q.b[k]);
            sm[q.c[k]] = t * q.id[k];
        };
        // the coarsest level in one warp's registers: pair t = row * hw + pr in
        // lane t; a cell's row neighbour is the lane's other cell on one side
        // and the next pair's on the other, the cells above and below are hw
        // lanes away
        auto coarsest_warp = [&](int l, const McPair<T>& q) {
            const int nx = P.nx[l], ny = P.ny[l], hw = (nx + 1) / 2;
            const int gj = row_of(l), pr = tid - gj * hw;
            const bool row = gj < ny;
            const int ls = gj > 0 ? lane - hw : (p.per_y ? lane + (ny - 1) * hw : -1);
            const int ln = gj < ny - 1 ? lane + hw : (p.per_y ? lane - (ny - 1) * hw : -1);
            // the neighbour outside the pair: west of an even column, east of an odd one
            const int lw = pr > 0 ? lane - 1 : (p.per_x ? lane + hw - 1 : -1);
            const int le = pr < hw - 1 ? lane + 1 : (p.per_x ? lane - (hw - 1) : -1);
            const T scale = P.scale[l];
            // a neighbour beyond a wall is added with factor 0: o + m x as one
            // fused operation rounds as o + x (m = 1) or gives o (m = 0)
            const T ms = ls < 0 ? T(0) : T(1), mn = ln < 0 ? T(0) : T(1);
            int lx[2];
            T mx[2], id[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                lx[k] = ((gj + k) & 1) ? le : lw;  // odd: the cell sits on an odd column
                mx[k] = lx[k] < 0 ? T(0) : T(1);
                id[k] = row ? q.id[k] : T(0);
            }
            T v[2] = {T(0), T(0)};  // red, black
            auto sweep = [&](int k, bool first) {
                T t = T(0);
                if (!first) {
                    const T o = v[1 - k];
                    const T x = __shfl_sync(0xffffffffu, o, lx[k] & 31);
                    const T s = __shfl_sync(0xffffffffu, o, ls & 31), n = __shfl_sync(0xffffffffu, o, ln & 31);
                    t = mg_fma(mx[k], x, o);
                    t = mg_fma(ms, s, t);
                    t = mg_fma(mn, n, t);
                }
                v[k] = mg_fma(scale, t, q.b[k]) * id[k];
            };
            // red first, then black first (a turned pair is two sweeps of one
            // colour in a row)
            sweep(0, true);
#pragma unroll 1
            for (int k = 1; k < MG_NC; ++k) {
                sweep(1, false);
                sweep(0, false);
            }
            sweep(1, false);
#pragma unroll 1
            for (int k = 0; k < MG_NC; ++k) {
                sweep(1, false);
                sweep(0, false);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if (q.in[k]) sm[q.c[k]] = v[k];
            __syncwarp();
        };
        // down; a warp without cells of a level waits for the way up at the
        // barrier of its last one
        int last = ns - 1;
        for (int l = ns; l < nlev; ++l) {
            const int n = (pairs_of(l) + 31) & ~31;
            if (tid >= n) break;
            last = l;
            const int bar = 1 + l - ns;
            McPair<T> q;
            make(l, q);
            const T scale = P.scale[l], ms = P.ms[l];
            if (l == nlev - 1) {
                if (n == 32 && !(P.nx[l] & 1)) {
                    coarsest_warp(l, q);
                    break;
                }
#pragma unroll 1
                for (int k = 0; k < MG_NC; ++k) {
                    half(q, 0, scale, k == 0);
                    mc_bar(bar, n);
                    half(q, 1, scale, false);
                    mc_bar(bar, n);
                }
#pragma unroll 1
                for (int k = 0; k < MG_NC; ++k) {
                    half(q, 1, scale, false);
                    mc_bar(bar, n);
                    half(q, 0, scale, false);
                    mc_bar(bar, n);
                }
                break;
            }
#pragma unroll 1
            for (int k = 0; k < MG_NU; ++k) {
                half(q, 0, scale, k == 0);
                mc_bar(bar, n);
                half(q, 1, scale, false);
                mc_bar(bar, n);
            }
            T* r = sm + P.tmp;  // r[c - xo]
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (!q.in[k]) continue;
                T ax = q.d[k] * sm[q.c[k]];
                ax = mg_fma(ms, sm[q.w[k]], ax);
                ax = mg_fma(ms, sm[q.e[k]], ax);
                ax = mg_fma(ms, sm[q.s[k]], ax);
                ax = mg_fma(ms, sm[q.n[k]], ax);
                r[q.c[k] - P.xo[l]] = q.b[k] - ax;
            }
            mc_bar(bar, n);
            // one coarse cell per thread: pair pr of row gj sits over coarse
            // column pr, so the even rows' threads take coarse row gj / 2
            const int nx = P.nx[l], ny = P.ny[l], sp = P.sp[l], nc = P.nx[l + 1], mc = P.ny[l + 1];
            const int gj = row_of(l), I = tid - gj * nc, J = gj >> 1;
            if (!(gj & 1) && J < mc) {
                T wx[4], wy[4];
                mc_rweights<T>(I, nc, p.per_x, p.bc[0], p.bc[2], wx);
                mc_rweights<T>(J, mc, p.per_y, p.bc[1], p.bc[3], wy);
                const int f = 2 * I;
                const int fa = f > 0 ? f - 1 : (p.per_x ? nx - 1 : 0), fd = f + 2 < nx ? f + 2 : (p.per_x ? 0 : nx - 1);
                T acc = T(0);
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    int g = 2 * J - 1 + a;
                    const bool out = g < 0 || g >= ny;
                    if (out) g = g < 0 ? g + ny : g - ny;
                    // (a cell beyond a wall has weight 0 and reads its neighbour)
                    const T* rr = r + (g + 1) * sp + PAD;
                    T rs = I > 0 || p.per_x ? mg_quarter(rr[fa]) : T(0);
                    rs = mg_fma(wx[1], rr[f], rs);
                    rs = mg_fma(wx[2], rr[f + 1], rs);
                    rs = mg_fma(wx[3], rr[fd], rs);
                    const T v = a == 0 ? mg_quarter(rs) : mg_fma(wy[a], rs, acc);
                    if (!out || p.per_y) acc = v;
                }
                sm[P.bo[l + 1] + J * P.sp[l + 1] + PAD + I] = mg_quarter(acc);
            }
            mc_bar(bar, n);
        }
        // up
        for (int l = last; l >= ns; --l) {
            if (l == nlev - 1) continue;
            const int n = (pairs_of(l) + 31) & ~31, bar = 1 + l - ns;
            const int nc = P.nx[l + 1], mc = P.ny[l + 1], csp = P.sp[l + 1];
            const int gj = row_of(l), pr = tid - gj * nc;  // (nx is even here: nc pairs per row)
            McPair<T> q;
            make(l, q);
            int J, NJ;
            T wyJ, wyN;
            mg_axis<T>(gj, mc, p.per_y, p.bc[1], p.bc[3], J, NJ, wyJ, wyN);
            const T wl = (pr == 0 && !p.per_x && p.bc[0] == 0) ? T(1) : T(0.75);
            const T wr = (pr == nc - 1 && !p.per_x && p.bc[2] == 0) ? T(1) : T(0.75);
            const T* cx = sm + P.xo[l + 1] + csp + PAD;  // row 0, column 0
            const int cw = pr > 0 ? pr - 1 : (p.per_x ? nc - 1 : -1), ce = pr < nc - 1 ? pr + 1 : (p.per_x ? 0 : nc);
            mc_bar(bar, n);  // the coarser level is done
            if (q.in[0] || q.in[1]) {
                const T* c0 = cx + J * csp;
                const T m0 = c0[pr];
                T v0 = wyJ * mg_fma(T(0.25), c0[cw], wl * m0), v1 = wyJ * mg_fma(T(0.25), c0[ce], wr * m0);
                if (NJ >= 0) {
                    const T* c1 = cx + NJ * csp;
                    const T m1 = c1[pr];
                    v0 = mg_fma(wyN, mg_fma(T(0.25), c1[cw], wl * m1), v0);
                    v1 = mg_fma(wyN, mg_fma(T(0.25), c1[ce], wr * m1), v1);
                }
                const int o = P.xo[l] + (gj + 1) * P.sp[l] + PAD + 2 * pr;
                sm[o] = sm[o] + v0;
                sm[o + 1] = sm[o + 1] + v1;
            }
            mc_bar(bar, n);
            const T scale = P.scale[l];
#pragma unroll 1
            for (int k = 0; k < MG_NU; ++k) {
                half(q, 1, scale, false);
                mc_bar(bar, n);
                half(q, 0, scale, false);
                mc_bar(bar, n);
            }
        }
        if (ns == 0) {
            __syncthreads();
            for (int g = warp; g < P.ny[0]; g += MC_WARPS)
                for (int i = lane; i < P.nx[0]; i += 32)
                    P.gx[(size_t)g * P.gpitch + i] = sm[P.xo[0] + (g + 1) * P.sp[0] + PAD + i];
        }
    }
    if (ns == 0) return;  // a single CTA
    // (CTA 0's last warps are free while its first ones solve)
    mc_pull(P, p, K, ns - 1, P.xo[ns - 1], 4, MC_WARPS - 8);
    mc_arrive();
    mc_wait();
    // ---- up, distributed levels
    for (int l = ns - 1; l >= 0; --l) {
        if (l + 1 < ns) {
            mc_pull(P, p, K, l + 1, P.bo[l + 1], 3, 0);
        } else {
            // level ns: the coarse rows of the band and three to each side, from CTA 0
            const int J0 = start[rank], J1 = start[rank + 1], csp = P.sp[ns];
            for (int J = J0 - 3 + warp; J < J1 + 3 && J0 < J1; J += MC_WARPS) {
                const int Jw = mg_dom(J, base, p.per_y);
                if (Jw < 0) continue;
                mc_row(sm + P.cxo + (J - J0 + MC_H) * csp, mc_map(sm + P.xo[ns] + (Jw + 1) * csp, 0u),
                       csp * (int)sizeof(T) / 16);
            }
        }
        // the last reads of other CTAs' memory: no CTA exits before all are done
        if (l == 0) mc_arrive();
        __syncthreads();
        switch (P.cpl[l]) {
            case 2: mc_up<T, 2, true>(P, p, K, l); break;
            case 4: mc_up<T, 4, true>(P, p, K, l); break;
            case -2: mc_up<T, 2, false>(P, p, K, l); break;
            case -4: mc_up<T, 4, false>(P, p, K, l); break;
            case 8:
                if constexpr (sizeof(T) == 4) mc_up<T, 8, true>(P, p, K, l);
                break;
            default:
                if constexpr (sizeof(T) == 4) mc_up<T, 8, false>(P, p, K, l);
        }
        if (l > 0) mc_arrive();
        mc_wait();
    }
}

// Shared-memory layout for levels lev[0 .. nlev) on C CTAs, ns = the first
// level CTA 0 takes alone; returns the bytes (0: a distributed level has more
// columns or a band more rows than its warps hold).  Fills the sizes and
// offsets.
template <typename T>
static size_t mg_coarse_layout(const MgLev<T>* lev, int nlev, int C, MgCoarse<T>* P) {
    constexpr int pad = McPad<T>::value;
    P->nlev = nlev;
    int ns = nlev - 1;
    for (int l = 0; l < nlev; ++l)
        if ((long long)lev[l].nx * lev[l].ny <= McMax<T>::alone) {
            ns = l;
            break;
        }
    P->ns = ns;
    const int rows = ns > 0 ? (lev[ns].ny + C - 1) / C : 0;  // band rows on level ns
    size_t o = 0, tmp = 0;
    for (int l = 0; l < nlev; ++l) {
        const int nx = lev[l].nx, ny = lev[l].ny;
        P->nx[l] = nx;
        P->ny[l] = ny;
        P->xo[l] = (int)o;
        if (l < ns) {
            const size_t n = (size_t)rows << (ns - l);
            if (nx > McMax<T>::columns || n + 2 * MC_H > MC_WARPS) return 0;
            const int cpl = nx <= 64 ? 2 : (nx <= 128 ? 4 : 8);
            P->cpl[l] = nx == 32 * cpl ? cpl : -cpl;
            P->sp[l] = 32 * cpl;
            o += (n + 2 * MC_H) * P->sp[l];
            P->bo[l] = (int)o;
            o += (n + 2 * MC_H) * P->sp[l];
            tmp = std::max(tmp, std::max((size_t)MC_WARPS * 16 * cpl, (n / 2 + 6) * 32 * cpl));  // row sums
        } else {
            P->sp[l] = (nx + 2 * pad + pad - 1) / pad * pad;
            P->inv[l] = (1u << 20) / (unsigned)((nx + 1) / 2) + 1u;
            o += (size_t)(ny + 2) * P->sp[l];
            P->bo[l] = (int)o;
            o += (size_t)ny * P->sp[l];
            tmp = std::max(tmp, (size_t)(ny + 2) * P->sp[l]);
        }
    }
    P->cxo = (int)o;
    if (ns > 0) o += (size_t)(rows + 2 * MC_H) * P->sp[ns];
    P->zero = (int)o;
    if (ns > 0) o += P->sp[0];
    P->tmp = (int)o;
    return (o + tmp) * sizeof(T);
}
