"""One V-cycle as a solve launches it (row windows, register strips, the cluster
launch and the levels its first block takes alone) against one launch per half
sweep, residual, restriction and prolongation on every level down to the coarsest;
FP64 also against the oracle.  The same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BCS = [((False, False), (0, 0, 0, 0)), ((True, True), (0, 0, 0, 0)), ((False, False), (0, 1, 1, 0)),
       ((True, False), (0, 1, 0, 0))]
# from hierarchies that one block solves alone (8 x 8 cells in one warp's registers,
# 17 x 9: an odd row) to distributed levels of 2, 4 and 8 columns to a lane and
# windows above them
SIZES = {"mixed": [(16, 16), (32, 16), (34, 18), (64, 32), (48, 80), (128, 128), (192, 96), (320, 256), (600, 304)],
         "fp64": [(16, 16), (32, 16), (34, 18), (48, 80), (64, 64), (112, 64), (256, 256)]}


@pytest.mark.parametrize("precision,nx,ny", [(p, *s) for p in SIZES for s in SIZES[p]])
@pytest.mark.parametrize("periodic,bc", BCS)
def test_vcycle_equals_levels(built, precision, nx, ny, periodic, bc):
    from cajitafluids_gb300 import Context
    from oracle import Oracle
    if (periodic[0] and nx % 4) or (periodic[1] and ny % 4):
        pytest.skip("a periodic axis of 34 or 18 cells has no coarser level")
    dt, rho = 0.01, 0.3
    r = np.random.default_rng(nx + 3 * ny).standard_normal((ny, nx))
    with Context(nx, ny, hi=(1.0, ny * (1.0 / nx)), periodic=periodic, precision=precision) as c:
        c.set_bc(bc)
        c.set_density(rho)
        z, rz = c.test_precondition(dt, r)
        zl, rzl = c.test_precondition(dt, r, levels=True)
    assert np.abs(z).max() > 0.0 and np.array_equal(z, zl)
    assert abs(rz - rzl) <= 1e-5 * abs(rzl)  # (FP32 products of another sum order)
    if precision == "fp64":
        zo, nlev = Oracle(nx, ny, hi=(1.0, ny / nx), periodic=periodic, bc=bc, density=rho, precon_mg=True).mg_apply(dt, r)
        assert nlev >= 2 and np.array_equal(z, zo)
