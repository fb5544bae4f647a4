"""The device-resident loop lets a mixed solve run to its iteration limit however
often the residual is replaced: with graphs on (the loop on the device, the solve on
chip or not) and off (polled by the host) the same iterations and the same bits."""
import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(16, 152), (96, 80), (1280, 1040)])  # the last one: launches, not on chip
@pytest.mark.parametrize("inner_tol,max_iter,max_outer", [(0.5, 300, 0), (0.7, 300, 0), (0.7, 300, 20)])
def test_mixed_jacobi_runs_to_its_limits(built, nx, ny, inner_tol, max_iter, max_outer):
    from cajitafluids_gb300 import Context
    rng = np.random.default_rng(nx)
    out = []
    u, v = rng.standard_normal((ny, nx)), rng.standard_normal((ny, nx))
    for graphs in (True, False):
        with Context(nx, ny, hi=(1.0, ny * (1.0 / nx)), periodic=(True, True), precision="mixed") as c:
            c.set_density(0.1)
            c.set_graphs(graphs)
            c.upload("u", u)
            c.upload("v", v)
            st = c.project(0.01, opts(tol=1e-13, max_iter=max_iter, precon="Diagonal", inner_tol=inner_tol,
                                      max_outer=max_outer))
            out.append((st, c.download("u"), c.download("v")))
    assert out[0][0] == out[1][0]
    st = out[0][0]
    # it ends converged or at one of the limits it was given
    assert st["status"] == 0 or st["iterations"] == max_iter or st["outer_iterations"] == (max_outer or 200)
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
