"""Read-backs and uploads of a D2Q9 solver on both sides of the sizes from which they
go through the staging ring."""
import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import Lbm2DConfig, WallKind, XBoundary, wall

pytestmark = pytest.mark.gpu

WEIGHTS = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)


def solver(nx, ny, storage):
    c = Lbm2DConfig(nx=nx, ny=ny, tau=0.6, x_boundary=XBoundary.periodic, bottom=wall(WallKind.periodic),
                    top=wall(WallKind.periodic))
    return S.make_gpu_solver(c, M.fluid_mask(nx, ny), storage=storage)


def fields(n):
    k = np.arange(n)
    return 1.0 + 1e-3 * np.sin(0.37 * k), 0.05 * np.cos(0.11 * k), 0.04 * np.sin(0.23 * k)


# 72 bytes a node: 1.5 MiB between 21,845 and 21,846 nodes.  The stored values are
# the binary64 ones rounded to binary32 of their distance (below 0.1) from the
# weight, formed with a few roundings of 2^-24 of sums below 0.5.
@pytest.mark.parametrize("size", [(5, 4369), (6, 3641), (400, 160)])
def test_binary32_populations(size):
    n = size[0] * size[1]
    one, two = solver(*size, "f32"), solver(*size, "f64")
    for s in (one, two):
        s.initialize(*fields(n))
    a, b = one.populations().reshape(9, n), two.populations().reshape(9, n)
    assert np.max(np.abs(a - b)) < 16 * 2.0 ** -24 * 0.5
    assert np.array_equal(np.float32(a - WEIGHTS[:, None]) + WEIGHTS[:, None], a)


# 24 bytes a node: 48 MiB from 2048 x 1024 nodes on.
@pytest.mark.parametrize("size", [(2047, 1024), (2048, 1024)])
@pytest.mark.parametrize("storage,eps", [("f32", 2.0 ** -24), ("f64", 2.0 ** -53)])
def test_initial_fields(size, storage, eps):
    n = size[0] * size[1]
    s = solver(*size, storage)
    state = fields(n)
    s.initialize(*state)
    m = s.macroscopic()
    # nine populations below 0.5, a few roundings each
    for got, want in zip((m.density, m.velocity_x, m.velocity_y), state):
        assert np.max(np.abs(got - want)) < 40 * eps
