"""The binary32 step on both sides of the size from which lattices run in linear
order (60,000 nodes), against the staged step's bits."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import Lbm3DConfig, Smagorinsky, WallKind, XBoundary, wall

pytestmark = pytest.mark.gpu


# Equal bits: the staged step runs the same node code, so no tolerance applies.
@pytest.mark.parametrize("sides,x_boundary", [(WallKind.slip, XBoundary.inflow_outflow),
                                              (WallKind.periodic, XBoundary.periodic)])
@pytest.mark.parametrize("size", [(129, 31, 15), (129, 31, 16), (65, 41, 40), (1000, 11, 10), (5, 145, 141)])
def test_same_bits_as_the_staged_step(size, sides, x_boundary):
    nx, ny, nz = size
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=x_boundary, outlet=Outlet.convective,
                    y_low=wall(sides), y_high=wall(sides), z_low=wall(sides), z_high=wall(sides), inlet_ux=0.04,
                    inlet_uy=0.002, smagorinsky=Smagorinsky(nx % 2 == 1, 0.1))
    mask = M.sphere_mask(nx, ny, nz, (nx / 2.0, 0.6, nz / 2.0), min(nx, ny, nz) / 4.0)
    state = W.noisy_state3d(c, mask, 5)
    populations = []
    for options in ({"kernel": "staged"}, {}, {"block_x": 32}, {"block_x": 96}, {"block_x": 256}):
        s = S.make_gpu_solver(c, mask, **options)
        s.initialize(*state)
        s.step(19)
        populations.append(s.populations())
        s.close()
    assert all(np.array_equal(p, populations[0]) for p in populations[1:])
