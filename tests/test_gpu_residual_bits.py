"""The mixed solver's residual cell by cell against the scalar double-float
operations in NumPy, the same bits: rows of 64 columns and their ends, an odd
width, the width that takes neither packed form, walls of both kinds and periodic
axes, units of one warp and of several."""
import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu

BCS = [((False, False), (0, 0, 0, 0)), ((True, True), (0, 0, 0, 0)), ((True, False), (0, 1, 0, 0)),
       ((False, True), (1, 0, 0, 0)), ((False, False), (0, 1, 1, 0))]
F = np.float32


def fma(a, b, c):
    """FP32 fused multiply-add: the product is exact in FP64, the sum is rounded to
    odd there, which makes the rounding to FP32 that follows the only one."""
    p = np.asarray(a, np.float64) * np.asarray(b, np.float64)
    c = np.broadcast_to(np.asarray(c, np.float64), p.shape)
    t = p + c
    bb = t - p
    err = (p - (t - bb)) + (c - bb)
    bits = t.copy().view(np.int64)
    inexact_even = (err != 0.0) & ((bits & 1) == 0)
    bits = np.where(inexact_even, np.where((err > 0.0) == (t > 0.0), bits + 1, bits - 1), bits)
    return bits.view(np.float64).astype(F)


def split(a):
    hi = a.astype(F)
    return hi, (a - hi.astype(np.float64)).astype(F)


def two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def quick(a, b):
    s = a + b
    return s, b - (s - a)


def add(x, y):  # accurate sum
    s, e = two_sum(x[0], y[0])
    th, tl = two_sum(x[1], y[1])
    s, e = quick(s, e + th)
    return quick(s, e + tl)


def add_s(x, y):
    s, e = two_sum(x[0], y[0])
    return quick(s, e + (x[1] + y[1]))


def mul(x, y):
    p = x[0] * y[0]
    e = fma(x[0], y[0], -p)
    e = fma(x[0], y[1], e)
    e = fma(x[1], y[0], e)
    return quick(p, e)


def neg(x):
    return -x[0], -x[1]


def _both(f, x):
    return f(x[0]), f(x[1])


def _residual(u, v, p, periodic, bc, scale, mscale):
    ny, nx = p.shape
    if periodic[0]:
        u = np.concatenate([u, u[:, :1]], axis=1)
    if periodic[1]:
        v = np.concatenate([v, v[:1]], axis=0)
    U, V, P = split(u), split(v), split(p)
    t = add(_both(lambda a: a[:, 1:], U), neg(_both(lambda a: a[:, :-1], U)))
    t = add(t, _both(lambda a: a[1:], V))
    t = add(t, neg(_both(lambda a: a[:-1], V)))
    b = mul(split(np.float64(mscale)), t)

    def ghosted(a):
        q = np.pad(a, 1)
        if periodic[0]:
            q[1:-1, 0], q[1:-1, -1] = a[:, -1], a[:, 0]
        if periodic[1]:
            q[0, 1:-1], q[-1, 1:-1] = a[-1], a[0]
        return q
    Q = _both(ghosted, P)
    d = np.full((ny, nx), 4.0, F)
    if not periodic[0]:
        d[:, 0] -= bc[0] == 0
        d[:, -1] -= bc[2] == 0
    if not periodic[1]:
        d[0] -= bc[1] == 0
        d[-1] -= bc[3] == 0
    nb = add_s(_both(lambda a: a[1:-1, :-2], Q), _both(lambda a: a[1:-1, 2:], Q))
    nb = add_s(nb, _both(lambda a: a[:-2, 1:-1], Q))
    nb = add_s(nb, _both(lambda a: a[2:, 1:-1], Q))
    t = add_s(mul((d, np.zeros_like(d)), P), neg(nb))
    return add_s(b, neg(mul(split(np.float64(scale)), t)))[0]


@pytest.mark.parametrize("nx,ny", [(64, 36), (126, 40), (129, 37), (130, 36), (192, 34), (516, 500)])
@pytest.mark.parametrize("periodic,bc", BCS)
def test_residual_bits(built, nx, ny, periodic, bc):
    from cajitafluids_gb300 import Context
    rng = np.random.default_rng(nx + ny)
    # (pairs hold 48 bits: values that are a pair come back as they went in)
    u, v = (np.float64(a[0]) + np.float64(a[1]) for a in
            (split(rng.standard_normal((ny, nx + (not periodic[0])))), split(rng.standard_normal((ny + (not periodic[1]), nx)))))
    if not periodic[0]:
        u[:, 0] = u[:, -1] = 0.0
    if not periodic[1]:
        v[0] = v[-1] = 0.0
    dt, rho, dx = 0.01, 0.3, 1.0 / nx
    with Context(nx, ny, hi=(1.0, ny * dx), periodic=periodic, precision="mixed") as c:
        dx = c.dx
        c.set_bc(bc)
        c.set_density(rho)
        c.upload("u", u)
        c.upload("v", v)
        # a pressure that leaves a residual small against b: the low parts show
        c.project(dt, opts(tol=1e-6, max_iter=20000, precon="Diagonal"))
        p = c.download("p")
        c.upload("u", u)
        c.upload("v", v)
        got = c.test_residual(dt)
        parts = c.test_residual(dt, split=True)
        assert np.array_equal(c.download("p"), p)
    want = _residual(u, v, p, periodic, bc, dt / ((rho * dx) * dx), -(1.0 / dx))
    assert 0.0 < np.abs(want).max() < 1e-3 * np.abs(u).max() / dx
    assert np.array_equal(got, want)
    assert np.array_equal(parts, want)
