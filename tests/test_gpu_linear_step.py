"""The linear-order step against the row kernel's node code: ragged rows, tiles
that end inside a row or beyond the lattice, lattices smaller than a tile."""
import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import (Lbm3DConfig, Outlet, Smagorinsky, SolidWall, Sponge, WallKind, XBoundary, wall)

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (9, 5, 4), (65, 7, 6), (64, 8, 5), (129, 11, 9), (40, 33, 17)]


def lattice(size, sides, x_boundary, solid_wall, les):
    nx, ny, nz = size
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=x_boundary, outlet=Outlet.convective,
                    y_low=wall(sides), y_high=wall(sides), z_low=wall(sides), z_high=wall(sides), inlet_ux=0.04,
                    inlet_uy=0.002, smagorinsky=Smagorinsky(les, 0.1), solid_wall=solid_wall,
                    sponge=Sponge(0.2, 2, 3, 1) if nx > 9 and x_boundary == XBoundary.inflow_outflow else Sponge())
    if nx < 9:
        mask = M.sphere_mask(nx, ny, nz, (1.0, 1.0, 1.0), 0.4 if x_boundary == XBoundary.periodic else -1.0)
    else:
        mask = M.sphere_mask(nx, ny, nz, (nx / 2.0, 0.6, nz / 2.0), min(ny, nz) / 2.6)
    return c, mask, W.noisy_state3d(c, mask, 5)


def populations(case, state, storage, **options):
    s = S.make_gpu_solver(*case, storage=storage, **options)
    s.initialize(*state)
    s.step(19)
    p = s.populations()
    s.close()
    return p


# Equal bits: the staged step (halfway walls) runs the same node code from row
# spans and the per-node row path, so no tolerance applies.
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("sides,x_boundary", [(WallKind.slip, XBoundary.inflow_outflow),
                                              (WallKind.periodic, XBoundary.periodic)])
@pytest.mark.parametrize("size", SIZES)
def test_same_bits_as_the_staged_step(size, sides, x_boundary, storage):
    c, mask, state = lattice(size, sides, x_boundary, SolidWall.halfway, size[1] % 2 == 1)
    want = populations((c, mask), state, storage, kernel="staged")
    for block in (0, 32, 96, 256):
        assert np.array_equal(populations((c, mask), state, storage, block_x=block), want)


# Interpolated walls take the row tiles for every storage; each against
# binary64 (itself equal to the oracle).  A population is below 0.4 and keeps 2^-24, 2^-11 or
# 2^-8 of its distance (below 0.04) from its weight; 19 steps, doubled for the
# collision's own rounding.
@pytest.mark.parametrize("storage,eps", [("f32", 2.0 ** -24), ("f16", 2.0 ** -11), ("bf16", 2.0 ** -8)])
@pytest.mark.parametrize("size", SIZES[1:])
def test_interpolated_walls_within_rounding(size, storage, eps):
    c, mask, state = lattice(size, WallKind.slip, XBoundary.inflow_outflow, SolidWall.interpolated, True)
    want = populations((c, mask), state, "f64")
    got = populations((c, mask), state, storage)
    assert np.max(np.abs(got - want)) < 19 * 2 * 0.04 * max(eps, 2.0 ** -22)


# The default tile changes at 5.5 million nodes: equal bits on both sides of it.
@pytest.mark.parametrize("nz,block", [(134, 128), (135, 256)])
def test_default_tile(nz, block):
    c, mask, _ = lattice((300, 136, nz), WallKind.slip, XBoundary.inflow_outflow, SolidWall.halfway, True)
    fields = []
    for options in ({}, {"block_x": 64}):
        s = S.make_gpu_solver(c, mask, storage="f16", **options)
        assert s.kernel_info()["block"] == options.get("block_x", block)
        s.step(5)
        m = s.macroscopic()
        fields.append([m.density, m.velocity_x, m.velocity_y, m.velocity_z])
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(*fields))
