"""Interpolated walls over one step, with a bound that the halfway rule exceeds: the
listed forms and the general node code between them (10,000, 300,000 and, for the
2-byte storages, 900,000 nodes)."""
import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.batch import CudaBatch3D
from orrery_b200.lbm3d import Lbm3DConfig, SolidWall, WallKind, XBoundary, wall

pytestmark = pytest.mark.gpu


# A stored population is off by at most half an ulp (2^-24, 2^-11 or 2^-9) of its
# distance from its weight: e.  The wall rules' weights add up to 1; the collision
# at tau 0.56 multiplies e by |1 - 1/tau| = 0.8 and adds 1/tau times the
# equilibrium's error, at most (19 e)/3 for the rest population: 12 e; then the
# result is rounded.  20 e leaves room for the terms of second order.  Binary32
# arithmetic adds some twenty roundings of 2^-24 of sums below 0.2.
@pytest.mark.parametrize("size", [(21, 20, 19), (21, 22, 23), (64, 32, 32), (83, 60, 60), (84, 61, 61), (129, 64, 40),
                                  (130, 84, 82), (131, 85, 83)])
@pytest.mark.parametrize("storage,half_ulp", [("f32", 2.0 ** -24), ("f16", 2.0 ** -11), ("bf16", 2.0 ** -9)])
def test_one_step_within_storage_rounding(size, storage, half_ulp):
    nx, ny, nz = size
    side = wall(WallKind.slip)
    mask = M.sphere_mask(nx, ny, nz, (nx / 2.1, ny / 2.2, nz / 1.9), min(ny, nz) / 2.6)

    def one_step(solid_wall, storage):
        c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=XBoundary.inflow_outflow, y_low=side, y_high=side,
                        z_low=side, z_high=side, inlet_ux=0.04, solid_wall=solid_wall)
        s = S.make_gpu_solver(c, mask, storage=storage)
        s.initialize(*W.noisy_state3d(c, mask, 5, amplitude=0.03))
        distance = np.max(np.abs(s.populations().reshape(19, -1) - WEIGHTS[:, None]))
        s.step(1)
        p = s.populations()
        s.close()
        return p, distance

    want, distance = one_step(SolidWall.interpolated, "f64")
    bound = 20 * half_ulp * distance + 20 * 2.0 ** -24 * 0.2
    assert np.max(np.abs(one_step(SolidWall.halfway, "f64")[0] - want)) > 4 * bound
    assert np.max(np.abs(one_step(SolidWall.interpolated, storage)[0] - want)) < bound


# Rest, 6 axes, 12 diagonals.
WEIGHTS = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


# A solver of this size takes the general node code (10,000 to 300,000 nodes) or the
# 64-register list, a member of a branched batch the list: the same bits.
@pytest.mark.parametrize("size", [(64, 32, 32), (129, 64, 40)])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_members_have_a_solvers_bits(size, storage):
    nx, ny, nz = size
    side = wall(WallKind.slip)
    mask = M.sphere_mask(nx, ny, nz, (nx / 2.1, ny / 2.2, nz / 1.9), min(ny, nz) / 2.6)
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.56, x_boundary=XBoundary.inflow_outflow, y_low=side, y_high=side,
                    z_low=side, z_high=side, inlet_ux=0.04, solid_wall=SolidWall.interpolated)
    alone, one, two = (S.make_gpu_solver(c, mask, storage=storage) for _ in range(3))
    batch = CudaBatch3D()
    for s in (one, two):
        batch.add(s)
    batch.set_schedule("rows", 128, branches=2)
    for n in (1, 18, 32):
        alone.step(n)
        batch.step(n)
        want = alone.populations()
        assert np.array_equal(one.populations(), want) and np.array_equal(two.populations(), want)
