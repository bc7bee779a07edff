"""The binary64 row step's default tile on ragged rows: one-warp blocks and
128-node tiles have equal bits, on both sides of the rule."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import Lbm3DConfig, Smagorinsky, SolidWall, WallKind, XBoundary, wall
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solid_wall", [SolidWall.halfway, SolidWall.interpolated])
@pytest.mark.parametrize("size,sides,block", [
    ((64, 24, 24), WallKind.slip, 128), ((64, 25, 24), WallKind.slip, 32), ((64, 25, 24), WallKind.no_slip, 128),
    ((65, 25, 24), WallKind.slip, 128), ((128, 30, 24), WallKind.slip, 128), ((129, 30, 24), WallKind.periodic, 32),
    ((224, 20, 20), WallKind.slip, 32), ((225, 20, 20), WallKind.slip, 128)])
def test_default_tile(size, sides, block, solid_wall):
    nx, ny, nz = size
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.55, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    y_low=wall(sides), y_high=wall(sides), z_low=wall(sides), z_high=wall(sides), inlet_ux=0.05,
                    solid_wall=solid_wall)
    mask = M.sphere_mask(nx, ny, nz, (nx / 3.0, ny / 2.2, nz / 2.0), ny / 5.0)
    got = []
    for options in ({}, {"block_x": 160 - block}):
        s = S.make_gpu_solver(c, mask, storage="f64", **options)
        assert s.kernel_info()["block"] == options.get("block_x", block)
        s.step(18)
        got.append(s.populations())
        s.close()
    assert np.array_equal(*got)


# The 96-register form (halfway walls, blocks up to 128, more than 2,368 warps
# of rows) and the plain one have the oracle's bits.
@pytest.mark.parametrize("size,block,dense", [((32, 74, 32), 0, False), ((32, 75, 32), 0, True), ((97, 25, 24), 128, True),
                                              ((97, 25, 24), 160, False), ((33, 37, 33), 96, True)])
@pytest.mark.parametrize("les", [False, True])
def test_dense_rows_match_the_oracle(size, block, dense, les):
    nx, ny, nz = size
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.55, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    y_low=wall(WallKind.slip), y_high=wall(WallKind.slip), z_low=wall(WallKind.periodic),
                    z_high=wall(WallKind.periodic), inlet_ux=0.05, smagorinsky=Smagorinsky(les, 0.1))
    mask = M.sphere_mask(nx, ny, nz, (nx / 3.0, 0.4, nz / 2.0), nz / 5.0)
    ref, s = O.Restated3D(c, mask.solid), S.make_gpu_solver(c, mask, storage="f64", block_x=block)
    assert (s.kernel_info()["registers"] <= 96) == dense
    ref.initialize()
    s.initialize()
    ref.step(19)
    s.step(19)
    assert np.array_equal(s.populations(), ref.populations())
