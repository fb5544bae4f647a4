"""The on-chip FP64 Jacobi-PCG's bounded grid barrier (the mixed one's:
test_gpu_errors.py).  With the test hook one block's first barrier waits for
arrivals that never come, with a short limit: it runs out, the launch records the
timeout and every block returns, the projection returns CF_ERR_TIMEOUT, and the
context then projects the same state to the bits of a fresh one."""
import numpy as np
import pytest

from cajitafluids_gb300 import CfError
from cajitafluids_gb300 import _lib as L
from helpers import load_state, make_pair, opts, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(60, 12), (256, 256), (1000, 1000)])  # one block, one unit a block, seven
def test_fp64_grid_barrier_timeout(built, nx, ny):
    lib = L.load()
    o, a = make_pair(nx, ny)
    b = make_pair(nx, ny)[1]
    st = random_state(o, np.random.default_rng(8), scale=0.1)
    so = opts(tol=1e-6, max_iter=200, precon="Diagonal")
    load_state(o, a, st)
    assert lib.cf_test_stall_wait(a.h, 1) == L.CF_OK
    try:
        with pytest.raises(CfError) as e:
            a.project(0.002, so)
        assert e.value.code == L.CF_ERR_TIMEOUT
        assert "timed out" in str(e.value)
    finally:
        lib.cf_test_stall_wait(a.h, 0)
    for f in ("q", "u", "v"):
        a.upload(f, st[f])
        b.upload(f, st[f])
    assert a.project(0.002, so) == b.project(0.002, so)
    for f in ("p", "u", "v"):
        assert np.array_equal(a.download(f), b.download(f)), f
