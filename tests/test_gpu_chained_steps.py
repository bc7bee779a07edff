"""Steps of one solver launched while the step before them ends: runs of every
length around a graph's, plain launches and graphs mixed, at lattices of less
than one wave and of several, give the populations of single steps."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import (Lbm2DConfig, Lbm3DConfig, SolidWall, WallKind, XBoundary, wall)

pytestmark = pytest.mark.gpu

OPEN, CLOSED = WallKind.slip, WallKind.no_slip


def lattice3(size, sides, solid_wall):
    nx, ny, nz = size
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.55, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    y_low=wall(sides), y_high=wall(sides), z_low=wall(sides), z_high=wall(sides), inlet_ux=0.05,
                    solid_wall=solid_wall)
    return c, M.sphere_mask(nx, ny, nz, (nx / 3.0, ny / 2.2, nz / 2.0), ny / 5.0)


def lattice2(size, sides):
    nx, ny = size
    c = Lbm2DConfig(nx=nx, ny=ny, tau=0.55, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    bottom=wall(sides), top=wall(sides), inlet_ux=0.05)
    return c, M.circle_mask(nx, ny, nx / 3.0, ny / 2.1, ny / 6.0)


CASES = ([lattice3(n, s, w) for n in ((17, 9, 9), (64, 32, 32), (128, 96, 64), (97, 65, 65))
          for s, w in ((OPEN, SolidWall.halfway), (OPEN, SolidWall.interpolated), (CLOSED, SolidWall.halfway))] +
         [lattice2(n, s) for n in ((17, 9), (400, 160), (2048, 512)) for s in (OPEN, CLOSED)])


# Equal bits: the order of the arithmetic does not depend on the launches.
@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
@pytest.mark.parametrize("k", range(len(CASES)))
def test_runs_equal_single_steps(k, storage):
    counts = (2, 15, 16, 17, 33, 3, 64)
    one, many = (S.make_gpu_solver(*CASES[k], storage=storage) for _ in range(2))
    for n in counts:
        for _ in range(n):
            one.step(1)
        many.step(n)
        assert np.array_equal(one.populations(), many.populations()), n
    one.close()
    many.close()
