"""The caller-owned-buffer D3Q19 step recorded into a CUDA graph: a replay uses
the inlet velocity of the recorded call, whatever the caller's structure and the
stack of the call hold by then."""
import ctypes

import numpy as np
import pytest

from orrery_b200 import masks as M
from orrery_b200._native import check, lib

pytestmark = pytest.mark.gpu

NX, NY, NZ = 24, 12, 10


class Params(ctypes.Structure):
    _fields_ = [("nx", ctypes.c_uint32), ("ny", ctypes.c_uint32), ("nz", ctypes.c_uint32),
                ("x_mode", ctypes.c_uint32), ("wall_kind", ctypes.c_uint32 * 4), ("wall_ux", ctypes.c_float * 4),
                ("inlet", ctypes.c_float * 3), ("tau", ctypes.c_float), ("smagorinsky_c2", ctypes.c_float),
                ("force", ctypes.c_float * 3), ("outlet_mode", ctypes.c_uint32), ("outlet_speed", ctypes.c_float),
                ("sponge_strength", ctypes.c_float), ("sponge_inlet", ctypes.c_uint32),
                ("sponge_outlet", ctypes.c_uint32), ("sponge_sides", ctypes.c_uint32),
                ("link_count", ctypes.c_uint32)]


def params(inlet):
    p = Params(nx=NX, ny=NY, nz=NZ, x_mode=1, tau=0.56, smagorinsky_c2=0.01, outlet_mode=0, outlet_speed=0.05,
               sponge_strength=0.2, sponge_inlet=3, sponge_outlet=4, sponge_sides=2)
    p.wall_kind[:] = [1, 1, 1, 1]
    p.inlet[:] = inlet
    return p


class Tables:
    """Tables and buffers of one lattice (populations at rest, history 0)."""

    def __init__(self, torch):
        mask = M.sphere_mask(NX, NY, NZ, (10.2, 6.1, 4.9), 2.6)
        codes = np.ascontiguousarray(1 - mask.solid.reshape(-1).astype(np.uint32))
        self.h = ctypes.c_void_p()
        check(lib().orr_gl3d_create(ctypes.byref(params((0.05, 0, 0))),
                                    codes.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), 0, ctypes.byref(self.h)),
              lib().orr_last_error)
        self.slack = int(lib().orr_gl3d_buffer_slack()) // 4
        n = 19 * NX * NY * NZ
        self.buffers = [torch.zeros(n + 2 * self.slack, device="cuda") for _ in range(2)]
        self.outlet = torch.zeros(5 * NY * NZ, device="cuda")

    def step(self, k, p, stream):
        at = [b.data_ptr() + 4 * self.slack for b in self.buffers]
        check(lib().orr_gl3d_step(self.h, ctypes.byref(p), at[k % 2], at[1 - k % 2], self.outlet.data_ptr(), None,
                                  stream), lib().orr_last_error)

    def close(self):
        lib().orr_gl3d_destroy(self.h)


INLETS = [(0.05, 0.002, -0.003), (0.04, -0.001, 0.006)]


def test_replay_uses_the_recorded_inlet():
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    plain, recorded = Tables(torch), Tables(torch)
    torch.cuda.synchronize()
    for k in range(4):
        plain.step(k, params(INLETS[k % 2]), stream.cuda_stream)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        for k in range(2):
            p = params(INLETS[k])
            recorded.step(k, p, torch.cuda.current_stream().cuda_stream)
            p.inlet[:] = [9.0, 9.0, 9.0]
    M.fluid_mask_3d(3, 3, 3)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(plain.buffers + [plain.outlet], recorded.buffers + [recorded.outlet]):
        assert torch.equal(a, b)
    del graph
    plain.close()
    recorded.close()
