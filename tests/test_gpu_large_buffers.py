"""The steps of the largest lattices.  Where 32-bit byte offsets do not reach a
buffer, a lattice of two equal halves along a periodic axis has the bits of one
half, whose step takes them."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import (Lbm2DConfig, Lbm3DConfig, Smagorinsky, WallKind, XBoundary, wall)

pytestmark = pytest.mark.gpu

LIMIT = 2 ** 32


def test_2d_offsets():
    nx, ny = 8192, 3650
    assert 9 * 8 * nx * ny < LIMIT - 8 * nx < LIMIT < 2 * 9 * 8 * nx * ny
    n = nx * ny
    half = M.fluid_mask(nx, ny).solid.reshape(ny, nx)
    half[1700:1760, 3000:3050] = 1
    half[:3, 5000:5007] = 1      # across the halves' border, and the lattice's ends
    fluid = half.reshape(-1) == 0
    state = [np.ones(n), np.where(fluid, 0.05 + W.uniform_noise(7, n, 0, 1e-3), 0.0),
             np.where(fluid, W.uniform_noise(7, n, 1, 1e-3), 0.0)]
    fields = []
    for halves in (1, 2):
        c = Lbm2DConfig(nx=nx, ny=ny * halves, tau=0.55, x_boundary=XBoundary.inflow_outflow,
                        outlet=Outlet.convective, bottom=wall(WallKind.periodic), top=wall(WallKind.periodic),
                        inlet_ux=0.05, inlet_uy=0.002, smagorinsky=Smagorinsky(True, 0.1))
        mask = M.SolidMask2D(nx, ny * halves, np.tile(half, (halves, 1)).reshape(-1))
        s = S.make_gpu_solver(c, mask, storage="f64")
        s.initialize(*(np.tile(f, halves) for f in state))
        s.step(19)
        m = s.macroscopic()
        fields.append([m.density, m.velocity_x, m.velocity_y])
        s.close()
    for one, two in zip(*fields):
        assert np.array_equal(two[:n], one) and np.array_equal(two[n:], one)


def test_two_byte_rows():
    nx, ny, nz = 512, 448, 248
    assert 19 * 2 * nx * ny * nz < LIMIT < 2 * 19 * 2 * nx * ny * nz
    n = nx * ny * nz
    half = np.zeros((nz, ny, nx), np.uint8)
    half[120:130, 200:230, 100:140] = 1
    half[:2, 440:, 250:253] = 1
    fields = []
    for halves in (1, 2):
        c = Lbm3DConfig(nx=nx, ny=ny, nz=nz * halves, tau=0.55, x_boundary=XBoundary.inflow_outflow,
                        outlet=Outlet.convective, y_low=wall(WallKind.slip), y_high=wall(WallKind.slip),
                        z_low=wall(WallKind.periodic), z_high=wall(WallKind.periodic), inlet_ux=0.05, inlet_uz=0.003,
                        smagorinsky=Smagorinsky(True, 0.1))
        mask = M.SolidMask3D(nx, ny, nz * halves, np.tile(half, (halves, 1, 1)).reshape(-1), None)
        s = S.make_gpu_solver(c, mask, storage="f16")
        s.step(13)
        m = s.macroscopic()
        fields.append([m.density, m.velocity_x, m.velocity_y, m.velocity_z])
        s.close()
    for one, two in zip(*fields):
        assert np.array_equal(two[:n], one) and np.array_equal(two[n:], one)


# Beyond 30 million nodes a 2-byte lattice runs in linear order with 256 threads and
# in rows with 128: the same bits.
def test_two_byte_rows_of_named_blocks():
    nx, ny, nz = 480, 260, 250
    assert nx * ny * nz > 30e6
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.55, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    y_low=wall(WallKind.slip), y_high=wall(WallKind.slip), z_low=wall(WallKind.slip),
                    z_high=wall(WallKind.slip), inlet_ux=0.05)
    mask = M.fluid_mask_3d(nx, ny, nz)
    mask.solid.reshape(nz, ny, nx)[100:120, 90:118, 100:133] = 1
    fields = []
    for block in (256, 128):
        s = S.make_gpu_solver(c, mask, storage="f16", block_x=block)
        s.step(13)
        m = s.macroscopic()
        fields.append([m.density, m.velocity_x, m.velocity_y, m.velocity_z])
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(*fields))
