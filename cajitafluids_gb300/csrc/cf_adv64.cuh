// FP64 advection pieces shared by the forward step and its adjoint: spline weights
// and the tables of what an entity's own coordinates fix.
#pragma once

#include "cf_internal.cuh"
#include "cf_mul64.cuh"

namespace cf {

static __constant__ double ENT_OFF_D[3][2] = {{0.5, 0.5}, {0.0, 0.5}, {0.5, 0.0}};

// a plain product on the integer pipes (IP) or by the hardware: the same bits
template <bool IP>
__device__ __forceinline__ double prod64(double a, double b) {
    return IP ? mul64i(a, b) : a * b;
}

// FP64 spline weights (Cajita B-spline order 1 / 3); the coordinate clamp, the cell
// and the linear weights come from the integer-pipe helpers (cf_internal.cuh).
template <int ORDER, bool IP = true>
__device__ __forceinline__ void weights64(double xi, int ext, int& k0, double* w) {
    int k;
    double t, s;
    if (ORDER == 1) {
        cell_fraction(clamp_bits(xi, 0.0, exact_double(ext - 1)), ext - 2, k, t, s);
        w[0] = s;
        w[1] = t;
        k0 = k;
    } else {
        cell_fraction(clamp_bits(xi, 1.0, exact_double(ext - 2)), ext - 3, k, t, s);
        double t2 = prod64<IP>(t, t);
        double t3 = prod64<IP>(t2, t);
        double s3 = prod64<IP>(prod64<IP>(s, s), s);
        w[0] = prod64<IP>(s3, 1.0 / 6.0);
        w[1] = fma(0.5, t3, -t2) + (2.0 / 3.0);
        w[2] = fma(0.5, (t + t2) - t3, 1.0 / 6.0);
        w[3] = prod64<IP>(t3, 1.0 / 6.0);
        k0 = k - 1;
    }
}

__device__ __forceinline__ double entity_coord(const Phys& p, int ent, int axis, int idx) {
    double t = exact_double(idx) + ENT_OFF_D[ent][axis];
    return p.gl[axis] + t * p.dx;
}

// What an entity's own coordinates fix depends on its column or its row alone:
// the coordinate, and the cells and weights of the first RK stage's samples of
// u and v.  Two warps
// work them out for the block's tile.
struct AdvAxis {
    double x0[32];
    double su[32], tu[32], sv[32], tv[32];
    int ku[32], kv[32];
    int u0, v0;  // every tu (tv) is zero: the samples sit on the grid's own points
};

// lane's entry of an axis table: the entity at local index idx along the axis, u and v
// extending to uext and vext (the whole warp calls)
__device__ __forceinline__ void fill_axis(AdvAxis& A, const Phys& p, int ent, int axis, int idx, int lane, int uext,
                                          int vext) {
    const double x = entity_coord(p, ent, axis, idx);
    double w[2];
    int k;
    A.x0[lane] = x;
    weights64<1>(times_rdx(x - p.low[E_FACEI][axis], p.rdx, p.rsh), uext, k, w);
    A.su[lane] = w[0];
    A.tu[lane] = w[1];
    A.ku[lane] = k;
    const bool u0 = __all_sync(0xffffffffu, w[1] == 0.0);
    weights64<1>(times_rdx(x - p.low[E_FACEJ][axis], p.rdx, p.rsh), vext, k, w);
    A.sv[lane] = w[0];
    A.tv[lane] = w[1];
    A.kv[lane] = k;
    const bool v0 = __all_sync(0xffffffffu, w[1] == 0.0);
    if (lane == 0) {
        A.u0 = u0;
        A.v0 = v0;
    }
}

}  // namespace cf
