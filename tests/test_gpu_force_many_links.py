"""Forces over more links than the force kernels' largest grid has threads."""
import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import Lbm2DConfig, Lbm3DConfig, WallKind, XBoundary, wall
from oracle import oracle as O

pytestmark = pytest.mark.gpu

THREADS = 148 * 8 * 256


def scattered(mask, share):
    mask.solid[:] = np.random.default_rng(5).random(mask.solid.size) < share
    mask.solid.reshape(-1, mask.nx)[:, [0, -1]] = 0  # the inlet and outlet columns must be fluid
    return mask


# Both sides add the same binary64 terms, the oracle one after another: the
# difference of two orders is at most 2 links eps sum|term|, and a term is at
# most 2 f (0.5 here at the most) times the arm.
def compare(s, ref, links, got_of, arm):
    assert links > THREADS
    ref.initialize()
    s.initialize()
    ref.step(1)
    s.step(1)
    got = [got_of(s.force()) for _ in range(3)]
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    assert np.all(np.abs(got[0] - np.asarray(ref.force())) <= 2 * links * 2.0**-53 * links * arm)
    s.close()


def test_force3d():
    nx, ny, nz = 128, 64, 64
    side = wall(WallKind.slip)
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.6, x_boundary=XBoundary.inflow_outflow, inlet_ux=0.03, inlet_uy=0.01,
                    y_low=side, y_high=side, z_low=side, z_high=side)
    mask = scattered(M.fluid_mask_3d(nx, ny, nz), 0.08)
    s = S.make_gpu_solver(c, mask, storage="f64")
    compare(s, O.Restated3D(c, mask.solid), len(s.links()[0]), lambda f: np.concatenate([f.force, f.moment]),
            np.array([1, 1, 1, nx, nx, nx]))


def test_force2d():
    nx, ny = 800, 400
    c = Lbm2DConfig(nx=nx, ny=ny, tau=0.6, x_boundary=XBoundary.inflow_outflow, inlet_ux=0.03, inlet_uy=0.01,
                    bottom=wall(WallKind.slip), top=wall(WallKind.slip))
    mask = scattered(M.fluid_mask(nx, ny), 0.2)
    s = S.make_gpu_solver(c, mask, storage="f64")
    compare(s, O.Restated2D(c, mask.solid), len(s.links()[0]), lambda f: np.array([f.x, f.y, f.moment]),
            np.array([1, 1, nx]))
