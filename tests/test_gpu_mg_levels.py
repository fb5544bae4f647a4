"""The row-per-warp multigrid level launches against the level-by-level
kernels, bit for bit: levels narrower than a window (112 | 120 columns, 22 | 24
rows), one cell pair short of and past its edges, several windows with a ragged
last one, and more windows than blocks; walls of both kinds and periodic axes."""
import numpy as np
import pytest

from test_gpu_mg_coarse import BCS, _project

pytestmark = pytest.mark.gpu

SIZES = {"mixed": [(32, 16), (112, 24), (116, 44), (120, 48), (244, 92), (600, 304), (2020, 940)],
         "fp64": [(272, 64), (224, 88), (228, 92), (240, 96), (244, 200), (600, 304), (1016, 1000),
                  # (two columns to a lane: 52 | 56 columns kept)
                  (104, 80), (106, 44), (112, 96), (114, 100), (156, 64), (192, 160), (256, 256)]}


@pytest.mark.parametrize("precision,nx,ny", [(p, *s) for p in SIZES for s in SIZES[p]])
@pytest.mark.parametrize("periodic,bc", BCS)
def test_level_rows_equal_levels(built, monkeypatch, precision, nx, ny, periodic, bc):
    rng = np.random.default_rng(nx + 5 * ny)
    u = rng.standard_normal((ny, nx + (not periodic[0])))
    v = rng.standard_normal((ny + (not periodic[1]), nx))
    if not periodic[0]:
        u[:, 0] = u[:, -1] = 0.0
    if not periodic[1]:
        v[0] = v[-1] = 0.0
    monkeypatch.setenv("CF_MG_RZ_FUSED", "0")  # (its sum order follows the tiling)
    sa, a = _project(nx, ny, precision, periodic, bc, {"u": u, "v": v})
    monkeypatch.setenv("CF_MG_FUSED", "0")
    sb, b = _project(nx, ny, precision, periodic, bc, {"u": u, "v": v})
    assert sa == sb
    for f in a:
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("periodic,bc", BCS)
def test_level_rows_rz(built, monkeypatch, periodic, bc):
    """r.z formed by the finest level's launch, and the ghosts it writes: CG
    converges as it does with r.z on its own."""
    nx, ny = 480, 256  # (coarsens far enough to converge in the 40 iterations)
    rng = np.random.default_rng(1)
    u = rng.standard_normal((ny, nx + (not periodic[0])))
    v = rng.standard_normal((ny + (not periodic[1]), nx))
    if not periodic[0]:
        u[:, 0] = u[:, -1] = 0.0
    if not periodic[1]:
        v[0] = v[-1] = 0.0
    sa, _ = _project(nx, ny, "mixed", periodic, bc, {"u": u, "v": v})
    monkeypatch.setenv("CF_MG_RZ_FUSED", "0")
    sb, _ = _project(nx, ny, "mixed", periodic, bc, {"u": u, "v": v})
    assert sa["status"] == 0 and sb["status"] == 0
    # a wrong r.z or ghost costs CG its conjugacy, which the count shows
    assert abs(sa["iterations"] - sb["iterations"]) <= 1
    assert max(sa["r_norm"], sb["r_norm"]) <= 1e-9 * sa["b_norm"]
