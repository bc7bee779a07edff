"""kernel_info's grid is the launch's: the row tiles, with the wall list's layers
where the step has them."""
import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import Lbm3DConfig, SolidWall, WallKind, XBoundary, wall

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,size,sides,listed", [
    ("f64", (97, 33, 20), WallKind.slip, True), ("f64", (97, 33, 20), WallKind.no_slip, False),
    ("f32", (128, 64, 64), WallKind.slip, True), ("f32", (64, 32, 32), WallKind.slip, False)])
def test_grid_counts_the_wall_list(storage, size, sides, listed):
    nx, ny, nz = size
    side = wall(sides)
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=XBoundary.inflow_outflow, y_low=side, y_high=side,
                    z_low=side, z_high=side, inlet_ux=0.04, solid_wall=SolidWall.interpolated)
    s = S.make_gpu_solver(c, M.sphere_mask(nx, ny, nz, (nx / 2.1, ny / 2.2, nz / 1.9), min(ny, nz) / 2.6),
                          storage=storage, block_x=32)
    layer = -(-nx // 32) * ny
    walls = len(np.unique(s.links()[0]))
    layers = -(-walls // (layer * 32)) if listed else 0
    assert s.kernel_info()["grid"] == layer * (nz + layers)
    s.close()
