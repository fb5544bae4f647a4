"""The FP64 adjoint of one advection over the reach a step may have: velocities of up
to 0.95 of a cell a step in every direction (each stencil start that a sample of each
kind can take), traces of exactly one cell, both orders, walls and periodic axes,
grids on and off the block size."""
import numpy as np
import pytest

from cajitafluids_gb300 import Context, SolverOptions
from cajitafluids_gb300 import _lib as L

pytestmark = pytest.mark.gpu

OPTS = SolverOptions(tol=1e-13, max_iter=20000)


def make(nx, ny, periodic):
    c = Context(nx, ny, lo=(0.0, 0.0), hi=(1.0, ny / nx), periodic=(periodic, periodic))
    c.set_density(0.1)
    c.set_quirks(L.CF_FIX_Q1)
    return c


def walls(c, u, v, periodic):
    if not periodic:
        u[:, 0] = u[:, -1] = 0.0
        v[0] = v[-1] = 0.0
    return u, v


@pytest.mark.parametrize("nx,ny", [(16, 8), (24, 20), (33, 31), (64, 40)])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("order", [1, 3])
def test_gradient_over_the_reach(built, nx, ny, periodic, order):
    c = make(nx, ny, periodic)
    rng = np.random.default_rng(nx * order + periodic)
    shape = {f: c.owned_shape(f) for f in ("q", "u", "v")}
    # a piecewise linear velocity has kinks at the cells' edges, and a central
    # difference that straddles one is off by the jump: with h = 1e-7 a step crosses
    # one in some 1e-3 of the runs.  Rounding: 1e-16 of sums of order 1e2 over h.
    q = rng.standard_normal(shape["q"])
    u, v = walls(c, rng.uniform(-1, 1, shape["u"]), rng.uniform(-1, 1, shape["v"]), periodic)
    dt = 0.95 / nx
    y = {f: rng.standard_normal(shape[f]) for f in shape}

    def loss(qq, uu, vv):
        for f, a in (("q", qq), ("u", uu), ("v", vv)):
            c.upload(f, a)
        c.forward_checkpointed(1, 1, dt, order, OPTS)
        return sum(float(np.sum(y[f] * c.download(f))) for f in y)

    loss(q, u, v)
    g = c.backward(y["q"], y["u"], y["v"])
    h = 1e-7
    d = {"q": rng.standard_normal(shape["q"])}
    d["u"], d["v"] = walls(c, rng.standard_normal(shape["u"]), rng.standard_normal(shape["v"]), periodic)
    for f in d:
        k = {e: (d[e] if e == f else 0.0) for e in d}
        fd = (loss(q + h * k["q"], u + h * k["u"], v + h * k["v"]) - loss(q - h * k["q"], u - h * k["u"], v - h * k["v"])) / (2 * h)
        an = float(np.sum(g[f] * d[f]))
        assert abs(fd - an) <= 2e-5 * np.sqrt(np.sum(g[f] ** 2) * np.sum(d[f] ** 2) / d[f].size) * np.sqrt(d[f].size), f
    c.close()


@pytest.mark.parametrize("direction", [(1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, -1)])
@pytest.mark.parametrize("order", [1, 3])
def test_one_whole_cell(built, direction, order):
    """A uniform flow of one cell a step moves q by one cell, and the adjoint back."""
    n = 32
    c = make(n, n, True)
    rng = np.random.default_rng(5)
    q, y = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    c.upload("q", q)
    c.upload("u", np.full((n, n), float(direction[0])))
    c.upload("v", np.full((n, n), float(direction[1])))
    c.forward_checkpointed(1, 1, 1.0 / n, order, OPTS)
    q1 = c.download("q")
    g = c.backward(y)
    lhs, rhs = float(np.sum(q1 * y)), float(np.sum(q * g["q"]))
    assert abs(lhs - rhs) <= 1e-12 * np.sum(np.abs(q1 * y))
    if order == 1:  # linear samples at the cells' centres: the shift itself
        assert np.allclose(g["q"], np.roll(y, (-direction[1], -direction[0]), (0, 1)), atol=1e-12)
    c.close()
