"""Which grids the Jacobi-PCG solves on chip, read from the kernels a projection
launches (fewer than its iterations on chip, two an iteration otherwise): up to eight
units of 64 x 16 cells (FP64) or four tiles of 128 x 16 (mixed) to an SM, as many as
shared memory or registers hold, and not one more; and the same bits as phase by
phase at the largest FP64 grid."""
import ctypes

import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu


def _sms():
    for name in ("libcudart.so", "libcudart.so.13", "libcudart.so.12"):
        try:
            rt = ctypes.CDLL(name)
        except OSError:
            continue
        n = ctypes.c_int(0)
        assert rt.cudaDeviceGetAttribute(ctypes.byref(n), 16, 0) == 0  # cudaDevAttrMultiProcessorCount
        return n.value
    raise RuntimeError("no CUDA runtime library")


def _project(nx, ny, precision, graphs=True):
    from cajitafluids_gb300 import Context
    rng = np.random.default_rng(nx + ny)
    with Context(nx, ny, hi=(1.0, ny * (1.0 / nx)), precision=precision) as c:
        c.set_density(0.3)
        c.set_graphs(graphs)
        u = rng.standard_normal(c.owned_shape("u"))
        v = rng.standard_normal(c.owned_shape("v"))
        u[:, 0] = u[:, -1] = 0.0
        v[0] = v[-1] = 0.0
        c.upload("u", u)
        c.upload("v", v)
        n = c.launches
        st = c.project(0.01, opts(tol=1e-12, max_iter=60, precon="Diagonal"))
        return st, c.launches - n, {f: c.download(f) for f in ("u", "v", "p")}


# the largest grid of 8 (4) columns of units (tiles) with at most that many to an SM
@pytest.mark.parametrize("per_sm,rows_more", [(1, 0), (2, 0), (4, 0), (7, 0), (8, 0), (8, 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_form_by_size(built, precision, per_sm, rows_more):
    across, limit = (8, 8) if precision == "fp64" else (4, 4)
    nx, ny = 512, 16 * (per_sm * _sms() // across + rows_more)
    st, launches, _ = _project(nx, ny, precision)
    assert st["iterations"] == 60
    if per_sm <= limit and not rows_more:
        assert launches < 60
    else:
        assert launches >= 120


def test_largest_fp64_grid_same_bits(built):
    nx, ny = 512, 16 * _sms() - 5
    a, la, fa = _project(nx, ny, "fp64")
    b, lb, fb = _project(nx, ny, "fp64", graphs=False)
    assert la < 60 and lb >= 120 and a == b
    for f in fa:
        assert np.array_equal(fa[f], fb[f]), f
