"""The on-chip Jacobi-PCG against the launch-per-phase kernels, bit for bit.

With graphs off every phase of the solve is a launch of its own; with graphs
on a grid whose vectors fit the SMs' shared memory is solved by one cooperative
launch per 512 iterations.  Sizes: one unit of 64 x 16 cells, its remainders,
one to seven units per block (grid sizes from the device's SM count), and a
solve longer than one launch."""
import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu


CASES = [
    # nx, ny, periodic, bc, max_iter
    (1, 1, (False, False), (0, 0, 0, 1), 10),
    (63, 15, (False, False), (0, 0, 0, 0), 200),
    (64, 16, (True, True), (0, 0, 0, 0), 200),
    (65, 17, (True, False), (1, 0, 0, 1), 200),
    (129, 33, (False, True), (0, 1, 1, 0), 200),
    (66, 130, (True, True), (0, 0, 0, 0), 600),
    (640, 240, (False, False), (0, 0, 0, 0), 60),    # 150 units: one per block
    (640, 250, (True, True), (0, 0, 0, 0), 60),      # 160 units: two
    (1000, 500, (False, False), (0, 0, 1, 0), 60),   # 512 units: four
    (1024, 1024, (True, False), (0, 0, 0, 0), 60),   # 1024 units: seven
    (1088, 1024, (False, True), (0, 0, 0, 0), 60),   # 1088 units: none (too large)
]
# tiles of 128 x 16 cells (mixed): one, two and four per block, five (too large)
MIXED = CASES[:6] + [(501, 333, (False, False), (0, 0, 0, 0), 0), (640, 250, (True, True), (0, 0, 0, 0), 0),
                     (1000, 500, (False, False), (0, 0, 1, 0), 0), (1024, 1024, (True, False), (0, 0, 0, 0), 0),
                     (1300, 1200, (False, False), (0, 1, 0, 0), 0)]


@pytest.mark.parametrize("nx,ny,periodic,bc,max_iter", CASES)
@pytest.mark.parametrize("solver", ["Diagonal", "None"])
def test_onchip_equals_launches(built, nx, ny, periodic, bc, max_iter, solver):
    from cajitafluids_gb300 import Context
    rng = np.random.default_rng(nx * 1000 + ny)
    out = []
    state = None
    for graphs in (True, False):
        c = Context(nx, ny, lo=(0.0, 0.0), hi=(1.0, ny * (1.0 / nx)), periodic=periodic)
        c.set_bc(bc)
        c.set_density(0.3)
        c.set_graphs(graphs)
        if state is None:
            state = {f: rng.standard_normal(c.owned_shape(f)) for f in ("q", "u", "v")}
            # no flow through the walls, as before every projection of a step
            if not periodic[0]:
                state["u"][:, 0] = state["u"][:, -1] = 0.0
            if not periodic[1]:
                state["v"][0] = state["v"][-1] = 0.0
        for f, a in state.items():
            c.upload(f, a)
        st = c.project(0.01, opts(tol=1e-12, max_iter=max_iter, precon=solver))
        out.append((st, {f: c.download(f) for f in ("u", "v", "p")}))
        c.close()
    assert out[0][0] == out[1][0]
    for f in ("u", "v", "p"):
        assert np.array_equal(out[0][1][f], out[1][1][f]), f


@pytest.mark.parametrize("nx,ny,periodic,bc,max_iter", MIXED)
def test_onchip_mixed(built, nx, ny, periodic, bc, max_iter):
    """The mixed solve's on-chip inner iteration (and, for the last size, the
    launch-per-phase one) against the FP64 solve: velocities to 1e-7 of the
    largest, the stated bound of a mixed projection, and the same bits with
    every phase of an iteration a launch of its own."""
    from cajitafluids_gb300 import Context
    from cajitafluids_gb300 import _lib as L
    rng = np.random.default_rng(nx * 1000 + ny + 1)
    out = []
    state = None
    for precision, graphs in (("fp64", True), ("mixed", True), ("mixed", False)):
        c = Context(nx, ny, lo=(0.0, 0.0), hi=(1.0, ny * (1.0 / nx)), periodic=periodic, precision=precision)
        c.set_bc(bc)
        c.set_density(0.3)
        c.set_quirks(L.CF_FIX_Q1)
        c.set_graphs(graphs)
        if state is None:
            state = {f: rng.standard_normal(c.owned_shape(f)) for f in ("u", "v")}
            if not periodic[0]:
                state["u"][:, 0] = state["u"][:, -1] = 0.0
            if not periodic[1]:
                state["v"][0] = state["v"][-1] = 0.0
        for f, a in state.items():
            c.upload(f, a)
        st = c.project(0.01, opts(tol=1e-9, max_iter=20000, precon="Diagonal"), raise_on_maxit=True)
        out.append((st, {f: c.download(f) for f in ("u", "v")}))
        c.close()
    for f in ("u", "v"):
        ref = out[0][1][f]
        assert np.abs(out[1][1][f] - ref).max() <= 1e-7 * max(np.abs(state[f]).max(), 1e-30), f
        assert np.array_equal(out[1][1][f], out[2][1][f]), f
    assert out[1][0] == out[2][0]


def test_onchip_many_launches(built):
    """A solve of more iterations than one launch takes, against the oracle."""
    from helpers import load_state, make_pair, random_state
    o, c = make_pair(200, 72, density=0.7)
    load_state(o, c, random_state(o, np.random.default_rng(5)))
    so = o.project(0.01, tol=1e-13, max_iter=5000)
    sg = c.project(0.01, opts(tol=1e-13, max_iter=5000, precon="Diagonal"))
    assert so["iterations"] > 512 and so["iterations"] == sg["iterations"]
    for f in ("u", "v", "p"):
        assert np.array_equal(o.get(f), c.download(f)), f
