"""The convective outlet's two history copies: a step reads the one beside its
source populations and writes the other, whatever the mix of single steps,
graphs, restarts and step kernels."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import WallKind, wall
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lattice(ny, sides):
    w = W.sphere3d(nx=48, ny=ny, nz=9, diameter=6.0, outlet=Outlet.convective)
    for name in ("y_low", "y_high", "z_low", "z_high"):
        setattr(w.config, name, wall(sides))
    return w


# The binary64 form has the oracle's bits (both evaluate the reference's
# expressions in its order), so the comparison is exact.
@pytest.mark.parametrize("ny", [7, 8, 17])
@pytest.mark.parametrize("sides,kernel", [(WallKind.slip, "rows"), (WallKind.slip, "staged"),
                                          (WallKind.no_slip, "rows")])
def test_history_follows_the_buffers(ny, sides, kernel):
    w = lattice(ny, sides)
    ref = O.Restated3D(w.config, w.mask.solid, w.mask.distance)
    s = S.make_gpu_solver(w.config, w.mask, storage="f64", kernel=kernel)
    for counts in ((1, 17, 16, 3), (2, 33)):     # the second run starts again from the odd buffer
        ref.initialize(w.rho, w.ux, w.uy, w.uz)
        s.initialize(w.rho, w.ux, w.uy, w.uz)
        for n in counts:
            ref.step(n)
            s.step(n)
        assert np.array_equal(s.populations(), ref.populations())
