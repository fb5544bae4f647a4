"""The mixed advection of large grids, whose CTAs take a tile's three entity kinds
together: a periodic field repeated over a large grid moves as the small one does
(one kind to a CTA there), bit for bit, with ragged last tiles, and staged windows
equal the global path with walls and inputs."""
import numpy as np
import pytest

from test_gpu_advect_staged import FIELDS, _pair, _same, _state
from cajitafluids_gb300 import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,reps", [(96, 80, 10), (70, 45, 16)])
@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("blob", [0.0, 6.0])
def test_repeated_field(built, nx, ny, reps, order, blob):
    s = _state(nx, ny, (True, True), seed=nx + order, blob=blob)
    umax = max(np.abs(s["u"]).max(), np.abs(s["v"]).max())
    dt = 0.5 / nx / (umax / (blob if blob else 1.0))
    out = []
    for r in (1, reps):
        c = Context(r * nx, r * ny, hi=(float(r), r * (ny / nx)), periodic=(True, True), precision="mixed")
        c.set_density(0.1)
        for f in FIELDS:
            c.upload(f, np.tile(s[f], (r, r)))
        c.advect(dt, order)
        out.append({f: c.download(f) for f in FIELDS})
        c.close()
    for f in FIELDS:
        assert np.array_equal(np.tile(out[0][f], (reps, reps)), out[1][f]), f


@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("blob", [0.0, 6.0])
def test_walls_equal_global_path(built, order, blob):
    nx, ny, periodic = 900, 811, (False, False)
    s = _state(nx, ny, periodic, seed=3, blob=blob)
    umax = max(np.abs(s["u"]).max(), np.abs(s["v"]).max())
    dt = 0.5 / nx / (umax / (blob if blob else 1.0))
    cs = _pair(nx, ny, periodic)
    for c in cs:
        for f in FIELDS:
            c.upload(f, s[f])
        c.advect(dt, order)
    _same(cs)
