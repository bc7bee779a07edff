"""Performance cases of the lattice Boltzmann solvers, through the package's
public entry points (``make_gpu_solver``, ``CudaBatch3D``, ``Server``,
``geometry``), and the same results in plain binary64 torch.

A case is a dict of plain values; its ``kind`` names the path:

  flow      one lattice (D3Q19, or D2Q9 when it has no ``nz``) from its initial
            state: steps with the force sampled every ``sample`` steps (the
            reference adapter's sampling), then the fields
  batch     lattices of different sizes advanced together, forces summed over
            the samples, then every lattice's fields
  serve     drag solves of different sizes submitted to a server together,
            each run for a fixed number of steps
  voxelize  a triangle mesh to solid flags and wall distances
"""
from __future__ import annotations

import math

import numpy as np
import torch

from orrery_b200 import geometry as G
from orrery_b200 import masks as M
from orrery_b200.batch import CudaBatch3D
from orrery_b200.lbm3d import (Lbm2DConfig, Lbm3DConfig, Outlet, Smagorinsky, SolidWall, Sponge, WallKind,
                               XBoundary, tau_of_viscosity, wall)
from orrery_b200.serve import Server
from orrery_b200.solver import make_gpu_solver
from orrery_b200.workloads import Workload3D

_STORAGE_BYTES = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}


def listed():
    return [
        # The smallest call: the lattice of the smoke run.  A step is a few
        # microseconds, so launches and the force read-back count.
        {"name": "sphere_64x32x32_f32", "kind": "flow", "nx": 64, "ny": 32, "nz": 32, "storage": "f32",
         "wall": "halfway", "outlet": "extrapolation", "sides": "slip", "les": 0.1, "sponge": False, "noise": False,
         "reynolds": 100.0, "u": 0.05, "body": 0.25, "aspect": 1.0, "steps": 200, "sample": 10},
        # The reference's D3Q19 GPU benchmark: 128^3 sphere channel with the
        # default (convective) outlet, BGK.
        {"name": "sphere_128_f32_convective", "kind": "flow", "nx": 128, "ny": 128, "nz": 128, "storage": "f32",
         "wall": "halfway", "outlet": "convective", "sides": "slip", "les": 0.0, "sponge": False, "noise": False,
         "reynolds": 300.0, "u": 0.05, "body": 0.1875, "aspect": 1.0, "steps": 200, "sample": 100},
        # The headline workload: 256 x 128 x 128 sphere, binary32, Smagorinsky,
        # started from noisy fields.
        {"name": "sphere_256x128x128_f32", "kind": "flow", "nx": 256, "ny": 128, "nz": 128, "storage": "f32",
         "wall": "halfway", "outlet": "extrapolation", "sides": "slip", "les": 0.1, "sponge": False, "noise": True,
         "reynolds": 200.0, "u": 0.05, "body": 0.25, "aspect": 1.0, "steps": 200, "sample": 10},
        # What the reference's adapter builds for a small body: interpolated
        # wall, convective outlet, absorbing layers, odd sizes.
        {"name": "adapter_97x65x65_f32", "kind": "flow", "nx": 97, "ny": 65, "nz": 65, "storage": "f32",
         "wall": "interpolated", "outlet": "convective", "sides": "slip", "les": 0.0, "sponge": True, "noise": False,
         "reynolds": 50.0, "u": 0.05, "body": 0.3, "aspect": 1.0, "steps": 200, "sample": 10},
        # The same for its Re 1000 validation lattice (12.5 M nodes).
        {"name": "adapter_337x193x193_f32", "kind": "flow", "nx": 337, "ny": 193, "nz": 193, "storage": "f32",
         "wall": "interpolated", "outlet": "convective", "sides": "slip", "les": 0.1, "sponge": True, "noise": False,
         "reynolds": 1000.0, "u": 0.05, "body": 0.25, "aspect": 1.0, "steps": 100, "sample": 10},
        # The precision form: 512 x 256 x 256 prolate ellipsoid in binary16.
        {"name": "ellipsoid_512x256x256_f16", "kind": "flow", "nx": 512, "ny": 256, "nz": 256, "storage": "f16",
         "wall": "halfway", "outlet": "extrapolation", "sides": "slip", "les": 0.12, "sponge": False, "noise": False,
         "reynolds": 1000.0, "u": 0.08, "body": 0.1875, "aspect": 2.0, "steps": 100, "sample": 10},
        # The binary64 form, which the other forms' errors are measured with.
        {"name": "sphere_128x64x64_f64", "kind": "flow", "nx": 128, "ny": 64, "nz": 64, "storage": "f64",
         "wall": "halfway", "outlet": "extrapolation", "sides": "slip", "les": 0.1, "sponge": False, "noise": False,
         "reynolds": 200.0, "u": 0.05, "body": 0.25, "aspect": 1.0, "steps": 200, "sample": 10},
        # D2Q9: the 400 x 160 cylinder (launch bound) and the reference's 2D
        # GPU benchmark.
        {"name": "cylinder_400x160_f32", "kind": "flow", "nx": 400, "ny": 160, "storage": "f32",
         "outlet": "extrapolation", "sides": "slip", "les": 0.1, "noise": True, "reynolds": 100.0, "u": 0.05,
         "body": 0.2, "steps": 1000, "sample": 50},
        {"name": "cylinder_2048x1024_f32", "kind": "flow", "nx": 2048, "ny": 1024, "storage": "f32",
         "outlet": "convective", "sides": "slip", "les": 0.0, "noise": False, "reynolds": 1000.0, "u": 0.05,
         "body": 0.0625, "steps": 500, "sample": 100},
        # The batched form: NACA wings on lattices between 96^3 and
        # 256 x 128 x 128, binary16.
        {"name": "batch_naca_8_f16", "kind": "batch", "count": 8, "low": 96, "high": 256, "storage": "f16",
         "les": 0.1, "steps": 200, "sample": 10},
        # The serving form: sphere-cone drag solves of different sizes, all
        # resident together.
        {"name": "serve_capsules_6_f16", "kind": "serve", "count": 6, "low": 64, "high": 192, "storage": "f16",
         "les": 0.1, "steps": 500, "window": 200},
        # A body's mask: the sphere-cone mesh on the adapter's grid.
        {"name": "voxelize_capsule_128x96x96", "kind": "voxelize", "nx": 128, "ny": 96, "nz": 96, "around": 96,
         "rings": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "flow", "flow2d", "flow2d", "batch", "serve", "voxelize"])
    if kind == "flow":
        storage = rng.choice(["f32", "f32", "f32", "f16", "f16", "bf16", "f64"])
        ny, nz = _log(rng, 32, 200), _log(rng, 32, 200)
        nx = _log(rng, max(48, max(ny, nz) // 2), 400)
        if rng.random() < 0.4:
            nx = max(48, nx // 16 * 16)
        adapter = rng.random() < 0.4
        wall_kind = "interpolated" if adapter else "halfway"
        steps = 20 * max(2, min(10, int(8e7 / (nx * ny * nz))))
        return {"kind": "flow", "nx": nx, "ny": ny, "nz": nz, "storage": storage, "wall": wall_kind,
                "outlet": "convective" if adapter or rng.random() < 0.4 else "extrapolation",
                "sides": "slip" if rng.random() < 0.75 else "periodic",
                "les": rng.choice([0.0, 0.1, 0.12]), "sponge": adapter, "noise": rng.random() < 0.3,
                "reynolds": round(math.exp(rng.uniform(math.log(50.0), math.log(500.0))), 3),
                "u": round(rng.uniform(0.03, 0.056), 4), "body": round(rng.uniform(0.18, 0.3), 4),
                "aspect": round(rng.uniform(1.0, 1.6), 3), "steps": steps, "sample": 10}
    if kind == "flow2d":
        nx, ny = _log(rng, 96, 2048), _log(rng, 64, 1024)
        return {"kind": "flow", "nx": nx, "ny": ny, "storage": rng.choice(["f32", "f32", "f32", "f64"]),
                "outlet": rng.choice(["convective", "extrapolation"]), "sides": rng.choice(["slip", "slip", "periodic"]),
                "les": rng.choice([0.0, 0.1]), "noise": rng.random() < 0.5,
                "reynolds": round(math.exp(rng.uniform(math.log(50.0), math.log(500.0))), 3),
                "u": round(rng.uniform(0.03, 0.056), 4), "body": round(rng.uniform(0.1, 0.25), 4),
                "steps": 300, "sample": 50}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 8), "low": 96, "high": rng.randint(128, 256),
                "storage": rng.choice(["f32", "f16", "f16", "bf16"]), "les": rng.choice([0.0, 0.1]),
                "steps": 20 * rng.randint(3, 10), "sample": 10}
    if kind == "serve":
        return {"kind": "serve", "count": rng.randint(2, 6), "low": 64, "high": rng.randint(80, 192),
                "storage": rng.choice(["f32", "f16"]), "les": 0.1, "steps": 100 * rng.randint(3, 5), "window": 200}
    nx = _log(rng, 48, 128)
    ny = rng.randint(40, 96)
    return {"kind": "voxelize", "nx": nx, "ny": ny, "nz": ny, "around": rng.randint(24, 96),
            "rings": rng.randint(6, 24)}


# ------------------------------------------------------------------ inputs --

def _ellipsoid(nx, ny, nz, centre, semi, angle):
    """Signed distance (first-order estimate, exact for a sphere) of an ellipsoid
    pitched about z, flat in the lattice order."""
    z, y, x = (np.arange(n, dtype=np.float64) - c for n, c in zip((nz, ny, nx), reversed(centre)))
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    ca, sa = math.cos(angle), math.sin(angle)
    k2 = ((ca * x + sa * y) / semi[0]) ** 2 + ((ca * y - sa * x) / semi[1]) ** 2
    return ((np.sqrt(k2 + (z / semi[2]) ** 2) - 1.0) * min(semi)).reshape(-1)


def _flow_inputs(case, seed):
    """Configuration, mask and initial fields (or None) of a flow case."""
    rng = np.random.default_rng([int(seed), 11])
    u = case["u"] * float(rng.uniform(0.92, 1.0))
    nx, ny = case["nx"], case["ny"]
    side = wall(WallKind.slip if case["sides"] == "slip" else WallKind.periodic)
    outlet = Outlet.convective if case["outlet"] == "convective" else Outlet.extrapolation
    les = Smagorinsky(case["les"] > 0.0, case["les"])
    shift = rng.uniform(-0.5, 0.5, 3)
    grow = float(rng.uniform(0.96, 1.04))
    if "nz" not in case:
        radius = 0.5 * case["body"] * ny * grow
        cfg = Lbm2DConfig(nx=nx, ny=ny, tau=tau_of_viscosity(u * 2.0 * radius / case["reynolds"]),
                          x_boundary=XBoundary.inflow_outflow, outlet=outlet, bottom=side, top=side, inlet_ux=u,
                          smagorinsky=les)
        mask = M.circle_mask(nx, ny, nx / 4.0 + shift[0], ny / 2.0 + shift[1], radius)
        fields = None
        if case["noise"]:
            fluid = mask.solid == 0
            fields = [np.ones(nx * ny)] + [np.where(fluid, v + rng.uniform(-1e-3, 1e-3, nx * ny), 0.0) for v in (u, 0.0)]
        return cfg, mask, fields
    nz = case["nz"]
    radius = 0.5 * case["body"] * min(ny, nz) * grow
    semi = (radius * case["aspect"], radius, radius)
    centre = (nx / 4.0 + shift[0], ny / 2.0 + shift[1], nz / 2.0 + shift[2])
    angle = math.radians(10.0) if case["aspect"] > 1.0 else 0.0
    d = _ellipsoid(nx, ny, nz, centre, semi, angle)
    inter = case["wall"] == "interpolated"
    mask = M.SolidMask3D(nx, ny, nz, (d <= 0.0).astype(np.uint8), d if inter else None)
    sponge = Sponge(0.1, nx // 12, nx // 8, min(ny, nz) // 16) if case["sponge"] else Sponge()
    cfg = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=tau_of_viscosity(u * 2.0 * semi[0] / case["reynolds"]),
                      x_boundary=XBoundary.inflow_outflow, outlet=outlet, y_low=side, y_high=side, z_low=side,
                      z_high=side, inlet_ux=u, smagorinsky=les, sponge=sponge,
                      solid_wall=SolidWall.interpolated if inter else SolidWall.halfway)
    fields = None
    if case["noise"]:
        n = nx * ny * nz
        fluid = mask.solid == 0
        fields = [np.ones(n)] + [np.where(fluid, v + rng.uniform(-1e-3, 1e-3, n), 0.0) for v in (u, 0.0, 0.0)]
    return cfg, mask, fields


def _batch_inputs(case, seed):
    """(configuration, mask) of every lattice of a batch."""
    rng = np.random.default_rng([int(seed), 12])
    sizes = np.random.default_rng([case["count"], case["high"]])  # the sizes are the case's, the bodies the seed's
    out = []
    for _ in range(case["count"]):
        nx = int(16 * round(sizes.uniform(case["low"], case["high"]) / 16.0))
        ny, nz = (int(round(sizes.uniform(96.0, 128.0))) for _ in range(2))
        u = 0.05 * float(rng.uniform(0.92, 1.0))
        chord = 0.4 * nx
        mask = M.naca_wing_mask(nx, ny, nz, str(rng.choice(["0012", "2412", "4415"])),
                                (0.25 * nx, 0.5 * ny, 0.5 * nz), chord, 0.6 * nz,
                                math.radians(float(rng.uniform(-4.0, 12.0))))
        cfg = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=tau_of_viscosity(u * chord / float(rng.uniform(200.0, 1000.0))),
                          x_boundary=XBoundary.inflow_outflow, outlet=Outlet.extrapolation,
                          y_low=wall(WallKind.slip), y_high=wall(WallKind.slip), z_low=wall(WallKind.slip),
                          z_high=wall(WallKind.slip), inlet_ux=u, smagorinsky=Smagorinsky(case["les"] > 0.0, case["les"]))
        out.append((cfg, mask))
    return out


def _serve_inputs(case, seed):
    """The workloads of a server's requests."""
    rng = np.random.default_rng([int(seed), 13])
    sizes = np.random.default_rng([case["count"], case["high"], 1])
    out = []
    for k in range(case["count"]):
        nx = int(16 * round(sizes.uniform(case["low"], case["high"]) / 16.0))
        ny = nz = int(round(64.0 + 0.375 * (nx - 64)))
        u = 0.05 * float(rng.uniform(0.92, 1.0))
        base = ny / 8.0
        mask = M.sphere_cone_mask(nx, ny, nz, (0.2 * nx, 0.5 * (ny - 1), 0.5 * (nz - 1)), base,
                                  math.radians(float(rng.uniform(20.0, 35.0))), base * float(rng.uniform(0.2, 0.4)))
        mask.distance = None
        cfg = Lbm3DConfig(nx=nx, ny=ny, nz=nz, tau=tau_of_viscosity(u * 2.0 * base / float(rng.uniform(100.0, 500.0))),
                          x_boundary=XBoundary.inflow_outflow, outlet=Outlet.extrapolation,
                          y_low=wall(WallKind.slip), y_high=wall(WallKind.slip), z_low=wall(WallKind.slip),
                          z_high=wall(WallKind.slip), inlet_ux=u, smagorinsky=Smagorinsky(True, case["les"]))
        out.append(Workload3D(f"capsule{k}", cfg, mask, None, None, None, None, 2.0 * base, math.pi * base * base))
    return out


def _mesh(case, seed):
    rng = np.random.default_rng([int(seed), 14])
    base = case["ny"] / 4.0 * float(rng.uniform(0.9, 1.0))
    mesh = G.sphere_cone_mesh(base, math.radians(float(rng.uniform(20.0, 35.0))), base * float(rng.uniform(0.2, 0.4)),
                              around=case["around"], nose_steps=case["rings"], cone_steps=case["rings"])
    shift = np.array([case["nx"] / 8.0, case["ny"] / 2.0, case["nz"] / 2.0]) + rng.uniform(-0.5, 0.5, 3)
    return G.TriangleMesh(mesh.vertices + shift, mesh.triangles), G.GridSpec((0.0, 0.0, 0.0), 1.0, case["nx"], case["ny"],
                                                                            case["nz"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flow":
        cfg, mask, fields = _flow_inputs(case, seed)
        solver = make_gpu_solver(cfg, mask, storage=case["storage"], allow_high_mach=case["u"] > 0.057)
        # A program that reads its fields again and again keeps their arrays.
        return {"case": case, "solver": solver, "fields": fields, "out": solver.macroscopic() if "nz" in case else None}
    if kind == "batch":
        batch, members = CudaBatch3D(), []
        for cfg, mask in _batch_inputs(case, seed):
            members.append(make_gpu_solver(cfg, mask, storage=case["storage"]))
            batch.add(members[-1])
        batch.set_schedule("rows", block=128, branches=64)
        return {"case": case, "batch": batch, "members": members, "out": [m.macroscopic() for m in members]}
    if kind == "serve":
        return {"case": case, "server": Server(storage=case["storage"], max_active=64, chunk_steps=100, sample_every=10),
                "requests": _serve_inputs(case, seed)}
    return {"case": case, "mesh": _mesh(case, seed)}


# --------------------------------------------------------------- one pass --

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flow":
        s = state["solver"]
        s.initialize(*(state["fields"] or ()))
        forces = []
        for _ in range(case["steps"] // case["sample"]):
            s.step(case["sample"])
            f = s.force()
            forces.append(np.concatenate([f.force, f.moment]) if "nz" in case else np.array([f.x, f.y, f.moment]))
        if "nz" not in case:
            m = s.macroscopic()
            return {"forces": np.array(forces), "fields": [m.density, m.velocity_x, m.velocity_y]}
        m = s.macroscopic(state["out"])
        return {"forces": np.array(forces), "fields": [m.density, m.velocity_x, m.velocity_y, m.velocity_z]}
    if kind == "batch":
        sums = state["batch"].step_sampled(case["steps"], case["sample"])
        fields = []
        for s, out in zip(state["members"], state["out"]):
            m = s.macroscopic(out)
            fields.append([m.density, m.velocity_x, m.velocity_y, m.velocity_z])
        return {"sums": sums, "fields": fields}
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(w, window=case["window"], max_steps=case["steps"], initial_state=False, fixed_steps=True)
               for w in state["requests"]]
        got = [server.wait(i) for i in ids]
        return {"coefficients": np.array([[r["cd"], r["cl"], r["cm"]] for r in got]),
                "forces": np.array([list(r["force"]) + list(r["moment"]) for r in got]),
                "steps": np.array([r["steps"] for r in got])}
    mesh, spec = state["mesh"]
    vox = G.voxelize(mesh, spec, winding=False)
    band = G.signed_distance_band(mesh, vox)
    return {"solid": vox.solid, "distance": band.distance, "in_band": band.in_band}


def _sizes(case):
    """Nodes of every lattice of a case."""
    if case["kind"] == "flow":
        return [case["nx"] * case["ny"] * case.get("nz", 1)]
    if case["kind"] == "batch":
        sizes = np.random.default_rng([case["count"], case["high"]])
        return [int(16 * round(sizes.uniform(case["low"], case["high"]) / 16.0)) *
                int(round(sizes.uniform(96.0, 128.0))) * int(round(sizes.uniform(96.0, 128.0)))
                for _ in range(case["count"])]
    sizes = np.random.default_rng([case["count"], case["high"], 1])
    nxs = [int(16 * round(sizes.uniform(case["low"], case["high"]) / 16.0)) for _ in range(case["count"])]
    return [nx * int(round(64.0 + 0.375 * (nx - 64))) ** 2 for nx in nxs]


def work(case):
    """Each step reads and writes every population once; a pass also writes the
    initial populations once and its fields.  About 250 operations a D3Q19 and
    110 a D2Q9 node update."""
    if case["kind"] == "voxelize":
        cells = case["nx"] * case["ny"] * case["nz"]
        triangles = 2 * case["around"] * (2 * case["rings"] + 1)
        return {"bytes": 10 * cells + 36 * triangles, "flops": 100 * cells * int(math.log2(triangles))}
    nodes = sum(_sizes(case))
    q = 19 if case["kind"] != "flow" or "nz" in case else 9
    values = q * _STORAGE_BYTES[case["storage"]]
    fields = 0 if case["kind"] == "serve" else 8 * (4 if q == 19 else 3)
    return {"bytes": nodes * (2 * values * case["steps"] + values + fields),
            "flops": nodes * case["steps"] * (250 if q == 19 else 110)}


# ------------------------------------------------- the same in binary64 torch --

_C3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
       (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
       (0, -1, 1)]
_C2 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]


class _Lattice:
    """Pull streaming and BGK collision on arrays of shape (nz, ny, nx): slip or
    periodic sides, regularized velocity inlet, zero-gradient or convective
    outlet, halfway or interpolated solid walls, Smagorinsky closure and
    absorbing layers."""

    def __init__(self, cfg, mask):
        self.cfg, self.dev = cfg, torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.flat = isinstance(cfg, Lbm2DConfig)
        self.c = _C2 if self.flat else _C3
        self.w = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4 if self.flat else [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
        self.shape = (1 if self.flat else cfg.nz, cfg.ny, cfg.nx)
        self.solid = torch.tensor(np.asarray(mask.solid) != 0, device=self.dev).reshape(self.shape)
        self.kinds = [(cfg.bottom if self.flat else cfg.y_low).kind,
                      WallKind.periodic if self.flat else cfg.z_low.kind]
        q = range(len(self.c))
        self.opp = [self.c.index(tuple(-v for v in self.c[i])) for i in q]
        self.mir = [[self.c.index(tuple(-v if a == axis else v for a, v in enumerate(self.c[i]))) for i in q]
                    for axis in (1, 2)]
        self.inlet = (cfg.inlet_ux, cfg.inlet_uy, 0.0 if self.flat else cfg.inlet_uz)
        ghost = self._padded(self.solid[None].expand(len(self.c), *self.shape).to(torch.uint8), False)
        self.links = []  # direction, node indices (z, y, x), wall fractions
        for i in q:
            at = (self._shifted(ghost, i) != 0) & ~self.solid
            z, y, x = torch.nonzero(at, as_tuple=True)
            if len(z):
                self.links.append((i, (z, y, x), self._fractions(mask, i, z, y, x)))
        self.sponge = None
        if not self.flat and cfg.sponge.strength > 0.0:
            best = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
            for axis, (lo, hi) in ((2, (cfg.sponge.inlet, cfg.sponge.outlet)), (1, (cfg.sponge.sides,) * 2),
                                   (0, (cfg.sponge.sides,) * 2)):
                if axis < 2 and self.kinds[1 - axis] == WallKind.periodic:
                    continue
                n = self.shape[axis]
                k = torch.arange(n, dtype=torch.float64, device=self.dev)
                view = [1, 1, 1]
                view[axis] = n
                for d, t in ((k, lo), (n - 1 - k, hi)):
                    if t:
                        best = torch.maximum(best, (((t - d) / t).clamp(min=0.0) ** 2).reshape(view))
            self.sponge = cfg.sponge.strength * best

    def _fractions(self, mask, i, z, y, x):
        q = torch.full(z.shape, 0.5, dtype=torch.float64, device=self.dev)
        if self.flat or self.cfg.solid_wall != SolidWall.interpolated:
            return q
        d = torch.tensor(mask.distance, dtype=torch.float64, device=self.dev).reshape(self.shape)
        size = torch.tensor(self.shape, device=self.dev)[:, None]
        here, step = torch.stack([z, y, x]), torch.tensor(self.c[i][::-1], device=self.dev)[:, None]
        inside = lambda p: ((p >= 0) & (p < size)).all(0)  # noqa: E731
        at = lambda a, p: a[tuple(torch.minimum(p.clamp(min=0), size - 1))]  # noqa: E731
        df, ds = at(d, here), at(d, here - step)
        good = inside(here - step) & (df >= 0) & (ds <= 0) & (df - ds > 0)
        frac = torch.where(good, (df / torch.where(good, df - ds, torch.ones_like(df))).clamp(max=1.0), q)
        blocked = ~inside(here + step) | at(self.solid, here + step)
        return torch.where((frac < 0.5) & blocked, q, frac)

    def _padded(self, f, inflow=True):
        """f with a ghost layer on every side: mirrored or periodic in y and z,
        the zero-gradient outlet (or nothing) in x."""
        p = torch.zeros((len(f),) + tuple(n + 2 for n in self.shape), dtype=f.dtype, device=self.dev)
        p[:, 1:-1, 1:-1, 1:-1] = f
        wrap, mir = self.kinds[0] == WallKind.periodic, self.mir[0]
        for i in range(len(f)):
            p[i, 1:-1, 0], p[i, 1:-1, -1] = (p[i, 1:-1, -2], p[i, 1:-1, 1]) if wrap else (p[mir[i], 1:-1, 1],
                                                                                      p[mir[i], 1:-1, -2])
        wrap, mir = self.kinds[1] == WallKind.periodic, self.mir[1]
        for i in range(len(f)):
            p[i, 0], p[i, -1] = (p[i, -2], p[i, 1]) if wrap else (p[mir[i], 1], p[mir[i], -2])
        if inflow:
            p[..., -1] = p[..., -2]
        return p

    def _shifted(self, p, i):
        x, y, z = self.c[i]
        nz, ny, nx = self.shape
        return p[i, 1 - z:1 - z + nz, 1 - y:1 - y + ny, 1 - x:1 - x + nx]

    def _feq(self, i, rho, u, uu):
        cu = sum(c * v for c, v in zip(self.c[i], u) if c) if any(self.c[i]) else 0.0
        return self.w[i] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * uu)

    def _pairs(self):
        return [(a, b) for a in range(3) for b in range(a, 3) if not (self.flat and b == 2)]

    def _moment2(self, neq):
        """Sum of c c neq by component."""
        return {(a, b): sum((self.c[i][a] * self.c[i][b]) * neq[i] for i in range(len(self.c))
                            if self.c[i][a] * self.c[i][b]) for a, b in self._pairs()}

    def initialize(self, fields):
        one = torch.ones(self.shape, dtype=torch.float64, device=self.dev)
        if fields is None:
            rho, u = one, [v * one for v in self.inlet]
        else:
            got = [torch.tensor(v, dtype=torch.float64, device=self.dev).reshape(self.shape) for v in fields]
            rho, u = got[0], got[1:] + ([0.0 * one] if self.flat else [])
        uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        self.f = torch.stack([torch.where(self.solid, self.w[i] * one, self._feq(i, rho, u, uu))
                              for i in range(len(self.c))])
        self.history = {i: self.f[i, ..., -1].clone() for i in range(len(self.c)) if self.c[i][0] < 0}

    def _reflected(self, i, at, q):
        z, y, x = at
        o = self.opp[i]
        nz, ny, nx = self.shape
        leaving = self.f[o, z, y, x]
        cx, cy, cz = self.c[i]
        farther = self.f[o, (z + cz).clamp(0, nz - 1), (y + cy).clamp(0, ny - 1), (x + cx).clamp(0, nx - 1)]
        return torch.where(q < 0.5, 2 * q * leaving + (1 - 2 * q) * farther,
                           (leaving + (2 * q - 1) * self.f[i, z, y, x]) / (2 * q))

    def _velocity_inlet(self, g):
        f = g[..., 0]
        ux, uy, _ = self.inlet
        known = sum((1 if c[0] == 0 else 2) * f[i] for i, c in enumerate(self.c) if c[0] <= 0)
        rho = known / (1.0 - ux)
        if self.flat:
            half = 0.5 * (f[2] - f[4])
            f[1] = f[3] + 2 / 3 * rho * ux
            f[5] = f[7] - half + rho * (ux / 6 + 0.5 * uy)
            f[8] = f[6] + half + rho * (ux / 6 - 0.5 * uy)
        else:
            for i, c in enumerate(self.c):
                if c[0] > 0:
                    f[i] = f[self.opp[i]] + 6 * self.w[i] * rho * sum(a * b for a, b in zip(c, self.inlet))
        uu = sum(v * v for v in self.inlet)
        feq = [self._feq(i, rho, self.inlet, uu) for i in range(len(self.c))]
        pi = self._moment2([f[i] - feq[i] for i in range(len(self.c))])
        for i, c in enumerate(self.c):
            f[i] = feq[i] + 4.5 * self.w[i] * sum((1 if a == b else 2) * (c[a] * c[b] - (1 / 3 if a == b else 0)) * v
                                                  for (a, b), v in pi.items())

    def step(self):
        cfg = self.cfg
        p = self._padded(self.f)
        g = torch.stack([self._shifted(p, i) for i in range(len(self.c))])
        del p
        for i, at, q in self.links:
            g[(i,) + at] = self._reflected(i, at, q)
        if cfg.outlet == Outlet.convective:
            for i, h in self.history.items():
                h.copy_((h + cfg.inlet_ux * g[i, ..., -1]) / (1.0 + cfg.inlet_ux))
                g[i, ..., -1] = h
        self._velocity_inlet(g)
        rho = g.sum(0)
        u = [sum(c[a] * g[i] for i, c in enumerate(self.c) if c[a]) / rho if not (self.flat and a == 2) else 0.0 * rho
             for a in range(3)]
        uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        tau = cfg.tau
        if cfg.smagorinsky.enabled:
            # sum c c f_eq = rho (I / 3 + u u)
            strain = 0.0
            for (a, b), v in self._moment2(g).items():
                v = v - rho * (u[a] * u[b] + (1 / 3 if a == b else 0.0))
                strain = strain + (1 if a == b else 2) * v * v
            k = 18.0 * math.sqrt(2.0) * cfg.smagorinsky.constant ** 2
            tau = 0.5 * (tau + torch.sqrt(tau * tau + k * torch.sqrt(strain) / rho))
        for i in range(len(self.c)):
            g[i] += (self._feq(i, rho, u, uu) - g[i]) / tau
            if self.sponge is not None:
                target = self._feq(i, 1.0, self.inlet, sum(v * v for v in self.inlet))
                g[i] += self.sponge * (target - g[i])
            g[i][self.solid] = self.w[i]
        self.f = g

    def force(self):
        """Momentum-exchange force and moment about the origin (2D: fx, fy, mz)."""
        total = torch.zeros(6, dtype=torch.float64, device=self.dev)
        for i, at, q in self.links:
            ex = self.f[(self.opp[i],) + at] + self._reflected(i, at, q)
            c = self.c[i]
            f = [-c[a] * ex for a in range(3)]
            r = [at[2 - a].double() - q * c[a] for a in range(3)]
            total += torch.stack([f[0].sum(), f[1].sum(), f[2].sum(), (r[1] * f[2] - r[2] * f[1]).sum(),
                                  (r[2] * f[0] - r[0] * f[2]).sum(), (r[0] * f[1] - r[1] * f[0]).sum()])
        total = total.cpu().numpy()
        return total[[0, 1, 5]] if self.flat else total

    def fields(self):
        rho = torch.where(self.solid, torch.ones_like(self.f[0]), self.f.sum(0))
        out = [rho] + [sum(c[a] * self.f[i] for i, c in enumerate(self.c) if c[a]) / rho
                       for a in range(2 if self.flat else 3)]
        return [torch.where(self.solid, torch.full_like(v, 1.0 if k == 0 else 0.0), v).reshape(-1).cpu().numpy()
                for k, v in enumerate(out)]


def _solve(cfg, mask, fields, steps, sample):
    lattice = _Lattice(cfg, mask)
    lattice.initialize(fields)
    forces = []
    for n in range(1, steps + 1):
        lattice.step()
        if n % sample == 0:
            forces.append(lattice.force())
    return np.array(forces), lattice.fields()


def _exact_distances(mesh, spec, band=3.0):
    """Closest-triangle distance of every cell centre, clamped to the band, with
    the sign of the summed solid angles."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    tri = torch.tensor(mesh.vertices[mesh.triangles.astype(np.int64)], device=dev)
    a, b, c = tri[:, 0], tri[:, 1], tri[:, 2]
    z, y, x = torch.meshgrid(*(torch.arange(n, dtype=torch.float64, device=dev) + 0.5 for n in (spec.nz, spec.ny, spec.nx)),
                             indexing="ij")
    points = torch.stack([x, y, z], -1).reshape(-1, 3)
    dot = lambda p, q: (p * q).sum(-1)  # noqa: E731
    normal = torch.linalg.cross(b - a, c - a)
    out = []
    for p in points.split(max(1, (1 << 23) // len(tri))):
        p = p[:, None, :]
        va, vb, vc = a - p, b - p, c - p
        la, lb, lc = va.norm(dim=-1), vb.norm(dim=-1), vc.norm(dim=-1)
        angle = 2.0 * torch.atan2(dot(va, torch.linalg.cross(vb, vc)),
                                  la * lb * lc + dot(va, vb) * lc + dot(vb, vc) * la + dot(vc, va) * lb)
        inside = angle.sum(-1) / (4.0 * math.pi) >= 0.5
        best = torch.full(la.shape, math.inf, dtype=torch.float64, device=dev)
        within = torch.ones_like(best, dtype=torch.bool)
        for s, t in ((a, b), (b, c), (c, a)):
            e = t - s
            k = (dot(p - s, e) / dot(e, e).clamp(min=1e-300)).clamp(0.0, 1.0)
            best = torch.minimum(best, (p - s - k[..., None] * e).norm(dim=-1))
            within &= dot(torch.linalg.cross(e.expand(p.shape[0], -1, -1), p - s), normal) >= 0.0
        height = dot(p - a, normal).abs() / normal.norm(dim=-1).clamp(min=1e-300)
        d = torch.where(within, torch.minimum(best, height), best).amin(-1).clamp(max=band)
        out.append(torch.where(inside, -d, d))
    return torch.cat(out).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "flow":
        cfg, mask, fields = _flow_inputs(case, seed)
        forces, got = _solve(cfg, mask, fields, case["steps"], case["sample"])
        return {"forces": forces, "fields": got}
    if kind == "batch":
        sums, fields = [], []
        for cfg, mask in _batch_inputs(case, seed):
            forces, got = _solve(cfg, mask, None, case["steps"], case["sample"])
            sums.append(forces.sum(0))
            fields.append(got)
        return {"sums": np.array(sums), "fields": fields}
    if kind == "serve":
        rows, means = [], []
        for w in _serve_inputs(case, seed):
            forces, _ = _solve(w.config, w.mask, None, case["steps"], 10)
            mean = forces[-(case["window"] // 10):].mean(0)
            q = 0.5 * w.config.inlet_ux ** 2 * w.reference_area
            rows.append([mean[0] / q, mean[1] / q, mean[5] / (q * w.reference_length)])
            means.append(mean)
        return {"coefficients": np.array(rows), "forces": np.array(means), "steps": None}
    mesh, spec = _mesh(case, seed)
    return {"solid": None, "distance": _exact_distances(mesh, spec), "in_band": None}
