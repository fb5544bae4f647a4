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
# windows above them; the last mixed one has register strips
SIZES = {"mixed": [(16, 16), (32, 16), (34, 18), (64, 32), (48, 80), (128, 128), (192, 96), (320, 256), (600, 304),
                   (2048, 1024)],
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


@pytest.mark.parametrize("seed", range(8))
def test_rz_holds_fp64s_bits(built, seed):
    """r.z of a finest level in row windows: terms of two cells eight rows apart in
    FP32 (r z + (r z), one rounding each), their sum no less precise than in FP64.  r is four cells of one
    row, 2^-24 and 2^-28 and 2^-32 times the first, so the sum has bits that a pair of
    FP32 values (48 bits) cannot hold."""
    from cajitafluids_gb300 import Context
    nx, ny = 240, 96
    rng = np.random.default_rng(seed)
    i, j = 4 * int(rng.integers(1, nx // 4 - 1)), int(rng.integers(0, ny))
    r = np.zeros((ny, nx))
    r[j, i:i + 4] = (rng.uniform(1.0, 2.0, 4) * 2.0 ** np.array([0.0, -24.0, -28.0, -32.0])).astype(np.float32)
    with Context(nx, ny, hi=(1.0, ny * (1.0 / nx)), precision="mixed") as c:
        z, rz = c.test_precondition(0.01, r)
    # the FP32 terms (the other cell of each unit holds r = 0), in exact arithmetic
    from fractions import Fraction
    terms = [Fraction(float(np.float32(r[j, k] * z[j, k]))) for k in range(i, i + 4)]  # (products of 48 bits are exact in FP64)
    exact = sum(terms)
    # at most three additions of non-zero terms, each off by half a unit of 2^-52
    assert abs(Fraction(rz) - exact) <= 3 * Fraction(1, 2 ** 53) * sum(abs(t) for t in terms)
