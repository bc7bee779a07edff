"""Lattices as deep as a grid's z holds, with interpolated walls on open sides: the
wall list's blocks fit beside the rows' or leave the step to the general node code."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import Lbm3DConfig, Smagorinsky, SolidWall, WallKind, XBoundary, wall
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# One layer of list blocks: 65,534 rows leave it room, 65,535 do not.  The
# binary64 form has the oracle's bits in both.
@pytest.mark.parametrize("nz", [65534, 65535])
def test_deep_lattices_match_the_oracle(nz):
    nx, ny = 9, 4
    side = wall(WallKind.slip)
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    y_low=side, y_high=side, z_low=side, z_high=side, inlet_ux=0.04,
                    smagorinsky=Smagorinsky(True, 0.1), solid_wall=SolidWall.interpolated)
    mask = M.sphere_mask(nx, ny, nz, (4.2, 1.6, nz - 2.3), 1.3)
    state = W.noisy_state3d(c, mask, 3)
    ref = O.Restated3D(c, mask.solid, mask.distance)
    s = S.make_gpu_solver(c, mask, storage="f64")
    ref.initialize(*state)
    s.initialize(*state)
    for n in (1, 18):
        ref.step(n)
        s.step(n)
    assert np.array_equal(s.populations(), ref.populations())
    s.close()
