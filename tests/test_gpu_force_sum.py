"""The force kernels' sum over blocks: one block, several, and more links than
the largest grid has threads; repeated calls on one solver."""
import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import Lbm2DConfig, Lbm3DConfig, WallKind, XBoundary, wall
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def scattered(mask, solids):
    cells = np.random.default_rng(solids).permutation(mask.solid.size)[:solids]
    mask.solid.reshape(-1)[cells] = 1
    mask.solid.reshape(-1, mask.nx)[:, [0, -1]] = 0  # the inlet and outlet columns must be fluid
    return mask


# Both sides add the same binary64 terms, the oracle one after another: the
# difference of two orders is at most 2 links eps sum|term|, and a term is at
# most 2 f (0.5 here at the most) times the arm.
@pytest.mark.parametrize("solids", [0, 1, 14, 15, 200, 7000])
def test_force3d(solids):
    nx, ny, nz = 64, 32, 32
    c = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=0.6, x_boundary=XBoundary.inflow_outflow, inlet_ux=0.03, inlet_uy=0.01,
                    y_low=wall(WallKind.slip), y_high=wall(WallKind.slip),
                    z_low=wall(WallKind.slip), z_high=wall(WallKind.slip))
    mask = scattered(M.fluid_mask_3d(nx, ny, nz), solids)
    ref, s = O.Restated3D(c, mask.solid), S.make_gpu_solver(c, mask, storage="f64")
    ref.initialize()
    s.initialize()
    links = 18 * solids
    for n in (1, 2):
        ref.step(n)
        s.step(n)
        want = np.asarray(ref.force())
        got = [np.concatenate([f.force, f.moment]) for f in (s.force() for _ in range(3))]
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
        bound = 2 * links * 2.0**-53 * links
        assert np.all(np.abs(got[0] - want) <= bound * np.array([1, 1, 1, nx, nx, nx]))
    s.close()


@pytest.mark.parametrize("solids", [0, 1, 30, 33, 400, 12000])
def test_force2d(solids):
    nx, ny = 400, 160
    c = Lbm2DConfig(nx=nx, ny=ny, tau=0.6, x_boundary=XBoundary.inflow_outflow, inlet_ux=0.03, inlet_uy=0.01,
                    bottom=wall(WallKind.slip), top=wall(WallKind.slip))
    mask = scattered(M.fluid_mask(nx, ny), solids)
    ref, s = O.Restated2D(c, mask.solid), S.make_gpu_solver(c, mask, storage="f64")
    ref.initialize()
    s.initialize()
    links = 8 * solids
    for n in (1, 2):
        ref.step(n)
        s.step(n)
        want = np.asarray(ref.force())
        got = [np.array([f.x, f.y, f.moment]) for f in (s.force() for _ in range(3))]
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
        bound = 2 * links * 2.0**-53 * links
        assert np.all(np.abs(got[0] - want) <= bound * np.array([1, 1, nx]))
    s.close()
