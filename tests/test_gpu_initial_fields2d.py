"""Initial fields of a D2Q9 solver whose storage has no room to stage them are
refused as an argument, with the reason."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import abi
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200.lbm3d import Lbm2DConfig, WallKind, XBoundary, wall

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_refusal_names_the_storage(storage):
    c = Lbm2DConfig(nx=64, ny=32, tau=0.6, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    bottom=wall(WallKind.slip), top=wall(WallKind.slip), inlet_ux=0.05)
    s = S.make_gpu_solver(c, M.fluid_mask(64, 32), storage=storage)
    n = 64 * 32
    with pytest.raises(S.LbmError, match="population storage of 4 or 8 bytes") as refused:
        s.initialize(np.ones(n), np.full(n, 0.05), np.zeros(n))
    assert refused.value.status == abi.ORR_ERR_INVALID
    s.close()
