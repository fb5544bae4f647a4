"""Point samples on both sides of the count from which their products run on the
integer pipes (65536): the oracle's bits on either."""
import numpy as np
import pytest

from helpers import load_state, make_pair, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 65535, 65536])
@pytest.mark.parametrize("order", [1, 3])
def test_interp_points_either_side(built, n, order):
    rng = np.random.default_rng(n + order)
    o, c = make_pair(40, 24)
    load_state(o, c, random_state(o, rng))
    o.fill_ghosts()
    c.fill_ghosts()
    xy = rng.uniform(-0.05, 1.05, (n, 2))
    for f in ("q", "u", "v"):
        assert np.array_equal(o.sample(f, order, xy), c.interp_points(f, order, xy)), f


@pytest.mark.parametrize("nx,ny", [(255, 257), (256, 256)])
def test_cell_velocity_either_side(built, nx, ny):
    rng = np.random.default_rng(nx)
    o, c = make_pair(nx, ny)
    load_state(o, c, random_state(o, rng))
    o.fill_ghosts()
    dx = 1.0 / nx
    x = -3.0 * dx + ((np.arange(nx) + 3).astype(np.float64) + 0.5) * dx
    y = -3.0 * dx + ((np.arange(ny) + 3).astype(np.float64) + 0.5) * dx
    xy = np.stack([a.ravel() for a in np.meshgrid(x, y)], axis=1)
    for f, got in zip(("u", "v"), c.cell_velocity()):
        assert np.array_equal(o.sample(f, 1, xy).reshape(ny, nx), got), f
