"""The mixed solver's residual against NumPy: b - A p formed from the downloaded
pressure, for row ends on and off a group of 64 columns, odd widths, walls of both
kinds and periodic axes, and for units of 4, 8 and 16 rows."""
import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu

BCS = [((False, False), (0, 0, 0, 0)), ((True, True), (0, 0, 0, 0)), ((True, False), (0, 1, 0, 0)),
       ((False, True), (1, 0, 0, 0)), ((False, False), (0, 1, 1, 0))]


@pytest.mark.parametrize("nx,ny", [(64, 36), (126, 40), (129, 37), (130, 36), (134, 52), (192, 34), (1028, 1012),
                                   (2050, 1280)])
@pytest.mark.parametrize("periodic,bc", BCS)
@pytest.mark.parametrize("inner_tol", [0.5, 1e-2])
def test_mixed_residual(built, nx, ny, periodic, bc, inner_tol):
    from cajitafluids_gb300 import Context
    if (periodic[0] and nx % 2) or (periodic[1] and ny % 2):
        pytest.skip("multigrid needs an even cell count along periodic axes")
    rng = np.random.default_rng(nx + ny)
    u = rng.standard_normal((ny, nx + (not periodic[0])))
    v = rng.standard_normal((ny + (not periodic[1]), nx))
    if not periodic[0]:
        u[:, 0] = u[:, -1] = 0.0
    if not periodic[1]:
        v[0] = v[-1] = 0.0
    dt, rho, dx = 0.01, 0.3, 1.0 / nx
    c = Context(nx, ny, lo=(0.0, 0.0), hi=(1.0, ny * dx), periodic=periodic, precision="mixed")
    c.set_bc(bc)
    c.set_density(rho)
    c.upload("u", u)
    c.upload("v", v)
    st = c.project(dt, opts(tol=1e-9, max_iter=3, precon="PFMG", inner_tol=inner_tol))
    p = c.download("p")
    c.close()

    ue = u if not periodic[0] else np.concatenate([u, u[:, :1]], axis=1)
    ve = v if not periodic[1] else np.concatenate([v, v[:1]], axis=0)
    b = -((ue[:, 1:] - ue[:, :-1]) + (ve[1:] - ve[:-1])) / dx
    assert abs(st["b_norm"] - np.linalg.norm(b)) <= 1e-6 * st["b_norm"]
    q = np.pad(p, 1)
    d = np.full((ny, nx), 4.0)
    if periodic[0]:
        q[1:-1, 0], q[1:-1, -1] = p[:, -1], p[:, 0]
    else:
        d[:, 0] -= bc[0] == 0
        d[:, -1] -= bc[2] == 0
    if periodic[1]:
        q[0, 1:-1], q[-1, 1:-1] = p[-1], p[0]
    else:
        d[0] -= bc[1] == 0
        d[-1] -= bc[3] == 0
    nb = q[1:-1, :-2] + q[1:-1, 2:] + q[:-2, 1:-1] + q[2:, 1:-1]
    r = np.linalg.norm(b - dt / (rho * dx * dx) * (d * p - nb))
    # r is stored in FP32 (6e-8 a cell) and summed in FP32 over a lane's rows (32
    # terms, 2e-6 at most); b itself is formed in double-float (2^-44 of terms that
    # are up to 1e4 times r after three iterations)
    assert abs(st["r_norm"] - r) <= 1e-5 * r
