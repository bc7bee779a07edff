"""The D2Q9 step in linear order: ragged rows, tiles across rows, every side and
edge rule, history copies over single steps and graphs, 64-bit offsets."""
import numpy as np
import pytest

from helpers import Outlet
from orrery_b200 import masks as M
from orrery_b200 import solver as S
from orrery_b200 import workloads as W
from orrery_b200.lbm3d import Lbm2DConfig, Smagorinsky, WallKind, XBoundary, wall
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lattice(size, sides, x_boundary, les, body=True):
    nx, ny = size
    speed = 0.01 if sides == WallKind.no_slip else 0.0
    c = Lbm2DConfig(nx=nx, ny=ny, tau=0.55, x_boundary=x_boundary, outlet=Outlet.convective,
                    bottom=wall(sides, speed), top=wall(sides, -speed), inlet_ux=0.05, inlet_uy=0.002,
                    smagorinsky=Smagorinsky(les, 0.1))
    # across the bottom side, and across the x edge of a periodic lattice
    x = 0.3 if x_boundary == XBoundary.periodic else nx / 2.0
    mask = M.circle_mask(nx, ny, x, 0.4, min(nx, ny) / 3.4) if body and nx > 8 else M.fluid_mask(nx, ny)
    n, fluid = nx * ny, mask.solid == 0
    state = (np.ones(n), np.where(fluid, 0.05 + W.uniform_noise(7, n, 0, 1e-3), 0.0),
             np.where(fluid, W.uniform_noise(7, n, 1, 1e-3), 0.0))
    return c, mask, state


# The binary64 form has the oracle's bits.
@pytest.mark.parametrize("size", [(3, 3), (9, 5), (65, 4), (128, 9), (131, 33)])
@pytest.mark.parametrize("sides,x_boundary", [(WallKind.slip, XBoundary.inflow_outflow),
                                              (WallKind.no_slip, XBoundary.inflow_outflow),
                                              (WallKind.periodic, XBoundary.periodic)])
def test_binary64_matches_the_oracle(size, sides, x_boundary):
    c, mask, state = lattice(size, sides, x_boundary, size[1] % 2 == 1)
    ref = O.Restated2D(c, mask.solid)
    for block in (0, 32, 256):
        s = S.make_gpu_solver(c, mask, storage="f64", block_x=block)
        for counts in ((1, 17, 3), (34,)):
            ref.initialize(*state)
            s.initialize(*state)
            for n in counts:
                ref.step(n)
                s.step(n)
            assert np.array_equal(s.populations(), ref.populations())


# A population (below 0.5) is rounded to 2^-24 of its distance from its weight
# (below 0.05) a few times a step: 21 steps, 8 roundings, one ulp of the sum.
@pytest.mark.parametrize("size", [(9, 5), (131, 33)])
def test_binary32_within_rounding(size):
    c, mask, state = lattice(size, WallKind.slip, XBoundary.inflow_outflow, True)
    ref = O.Restated2D(c, mask.solid)
    s = S.make_gpu_solver(c, mask)
    ref.initialize(*state)
    s.initialize(*state)
    ref.step(21)
    s.step(21)
    assert np.max(np.abs(s.populations() - ref.populations())) < 21 * 8 * 2.0 ** -22 * 0.05


# Buffers above 4 GB take 64-bit offsets; a uniform stream stays uniform.
def test_64_bit_offsets_keep_a_uniform_stream():
    c, mask, _ = lattice((8192, 7300), WallKind.slip, XBoundary.inflow_outflow, False, body=False)
    c.inlet_uy = 0.0
    s = S.make_gpu_solver(c, mask, storage="f64")
    s.step(18)
    m = s.macroscopic()
    assert np.max(np.abs(m.density - 1.0)) < 1e-13
    assert np.max(np.abs(m.velocity_x - 0.05)) < 1e-13
    assert np.max(np.abs(m.velocity_y)) < 1e-13


# Initial fields are staged in a population buffer, which the 2-byte storages
# have no room for: refused before the copy, direct or through the ring, and
# the solver keeps its state.
@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("size", [(64, 32), (2048, 1024)])
def test_two_byte_storages_refuse_initial_fields(size, storage):
    nx, ny = size
    c = Lbm2DConfig(nx=nx, ny=ny, tau=0.6, x_boundary=XBoundary.inflow_outflow, outlet=Outlet.convective,
                    bottom=wall(WallKind.slip), top=wall(WallKind.slip), inlet_ux=0.05)
    s = S.make_gpu_solver(c, M.fluid_mask(nx, ny), storage=storage)
    s.step(3)
    before = s.populations()
    n = nx * ny
    with pytest.raises(S.LbmError):
        s.initialize(np.ones(n), np.full(n, 0.05), np.zeros(n))
    assert np.array_equal(s.populations(), before)
    s.step(17)
    assert np.all(np.isfinite(s.populations()))
