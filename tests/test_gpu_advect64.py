"""The FP64 advection's integer-pipe coordinates and per-axis tables against
the oracle, bit for bit: tall and flat tiles, power-of-two and other cell
sizes, traces that end on grid points or past the clamps, and taps that are
not finite."""
import numpy as np
import pytest

from helpers import assert_fields_equal, load_state, make_pair, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,periodic", [(33, 29, (False, False)), (64, 40, (True, True)), (128, 128, (False, True)),
                                            (700, 650, (False, False)), (640, 704, (True, False))])
@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("flow", ["random", "still", "cells", "far"])
def test_advect64_bitwise(built, nx, ny, periodic, order, flow):
    o, c = make_pair(nx, ny, periodic=periodic, body=(0.5, -1.0))
    st = random_state(o, np.random.default_rng(nx + order))
    dx = 1.0 / nx
    dt = 0.25 * dx
    if flow == "still":
        st["u"][:] = 0.0
        st["v"][:] = -0.0
    elif flow == "cells":  # half and whole cells a step
        st["u"][:] = 2.0
        st["v"][:] = -4.0
    elif flow == "far":    # past the ends of the ghosted arrays
        st["u"] *= 40.0
        st["v"] *= 4.0e6
    load_state(o, c, st)
    for _ in range(2):
        o.advect(dt, order)
        c.advect(dt, order)
    assert_fields_equal(o, c, tag=flow)


@pytest.mark.parametrize("order", [1, 3])
def test_advect64_not_finite(built, order):
    n = 64
    o, c = make_pair(n, n)
    st = random_state(o, np.random.default_rng(3), scale=0.2)
    for f in ("q", "u", "v"):
        st[f][20, 30] = np.inf
        st[f][40, 10] = np.nan
        st[f][5, 50] = -np.inf
    load_state(o, c, st)
    o.advect(0.2 / n, order)
    c.advect(0.2 / n, order)
    for f in ("q", "u", "v"):
        assert np.array_equal(o.get(f), c.download(f), equal_nan=True), f
