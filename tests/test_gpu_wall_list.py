"""Interpolated walls on open lattices: the boundary nodes are stepped from
their list.  Bodies that cross the sides and (periodic x) the x edges put
listed nodes on face rows, in corners and at the row ends."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import (Lbm3DConfig, Smagorinsky, SolidWall, Sponge, WallKind, XBoundary, wall)
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lattice(sides, x_boundary, size, centre, radius, sponge=False):
    nx, ny, nz = size
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=x_boundary, outlet=Outlet.convective,
                    y_low=wall(sides), y_high=wall(sides), z_low=wall(sides), z_high=wall(sides), inlet_ux=0.04,
                    inlet_uy=0.003, inlet_uz=-0.002, smagorinsky=Smagorinsky(True, 0.1),
                    solid_wall=SolidWall.interpolated, sponge=Sponge(0.3, 3, 4, 2) if sponge else Sponge())
    mask = M.sphere_mask(nx, ny, nz, centre, radius)
    return c, mask, W.noisy_state3d(c, mask, 3)


CASES = {
    "few": ((9, 7, 5), (4.3, 3.1, 2.2), 0.6),            # fewer boundary nodes than one block
    "face": ((33, 17, 12), (14.2, 1.4, 9.7), 4.3),       # across a y side and near a z side
    "corner": ((130, 24, 23), (60.1, 0.3, 22.2), 7.7),   # across a y and a z side; ragged row tiles
    "many": ((64, 40, 40), (30.3, 20.2, 19.6), 15.4),    # several blocks of boundary nodes
}


# The binary64 form has the oracle's bits.
@pytest.mark.parametrize("sides", [WallKind.slip, WallKind.periodic])
@pytest.mark.parametrize("name", sorted(CASES))
def test_boundary_nodes_match_the_oracle(name, sides):
    size, centre, radius = CASES[name]
    c, mask, state = lattice(sides, XBoundary.inflow_outflow, size, centre, radius, sponge=name == "many")
    ref = O.Restated3D(c, mask.solid, mask.distance)
    s = S.make_gpu_solver(c, mask, storage="f64")
    ref.initialize(*state)
    s.initialize(*state)
    ref.step(19)
    s.step(19)
    assert np.array_equal(s.populations(), ref.populations())


def test_periodic_x_edges_match_the_oracle():
    c, mask, state = lattice(WallKind.periodic, XBoundary.periodic, (31, 14, 13), (0.4, 6.8, 6.3), 4.2)
    ref = O.Restated3D(c, mask.solid, mask.distance)
    s = S.make_gpu_solver(c, mask, storage="f64")
    ref.initialize(*state)
    s.initialize(*state)
    ref.step(19)
    s.step(19)
    assert np.array_equal(s.populations(), ref.populations())


# Binary32 rounds each population to 6e-8 of its O(0.1) size a few times a
# step; 19 steps stay far within the 1e-5 relative bar of the full-size runs.
def test_binary32_boundary_nodes():
    c, mask, state = lattice(WallKind.slip, XBoundary.inflow_outflow, *CASES["corner"], sponge=True)
    ref = O.Restated3D(c, mask.solid, mask.distance)
    s = S.make_gpu_solver(c, mask)
    ref.initialize(*state)
    s.initialize(*state)
    s.set_inlet_velocity((0.03, -0.001, 0.002))
    ref.set_inlet_velocity((0.03, -0.001, 0.002))
    ref.step(19)
    s.step(19)
    a, b = s.populations(), ref.populations()
    assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-5
