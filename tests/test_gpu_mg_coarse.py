"""The cluster launch of the coarse multigrid levels against the
level-by-level kernels, bit for bit: every first level it takes (32 lanes of 2,
4 and 8 columns, filled and not), walls of both kinds and periodic axes."""
import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu

BCS = [((False, False), (0, 0, 0, 0)), ((True, True), (0, 0, 0, 0)), ((True, False), (0, 1, 0, 0)),
       ((False, True), (1, 0, 0, 0)), ((False, False), (0, 1, 1, 0))]
# the finest FP32 level stays a tile launch: the cluster starts at half the size
SIZES = {"mixed": [(512, 512), (320, 256), (256, 128), (192, 96), (128, 128), (96, 64), (64, 32)],
         "fp64": [(256, 256), (128, 128), (96, 112), (112, 64), (64, 64), (48, 80), (32, 16), (16, 16)]}


def _project(nx, ny, precision, periodic, bc, state):
    from cajitafluids_gb300 import Context
    c = Context(nx, ny, lo=(0.0, 0.0), hi=(1.0, ny * (1.0 / nx)), periodic=periodic, precision=precision)
    c.set_bc(bc)
    c.set_density(0.3)
    for f in ("u", "v"):
        c.upload(f, state[f])
    st = c.project(0.01, opts(tol=1e-9, max_iter=40, precon="PFMG"))
    out = {f: c.download(f) for f in ("u", "v", "p")}
    c.close()
    return st, out


@pytest.mark.parametrize("precision,nx,ny", [(p, *s) for p in SIZES for s in SIZES[p]])
@pytest.mark.parametrize("periodic,bc", BCS)
def test_coarse_cluster_equals_levels(built, monkeypatch, precision, nx, ny, periodic, bc):
    rng = np.random.default_rng(nx + 7 * ny)
    # (owned shapes: one face more along a walled axis, none of them with flow)
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
