"""What a user of the engine has it do, as measurable cases.

A case is one pass of a user's program over the public entry points: advance a
flow and read its fields, follow it with monitors, set a lattice up from a
surface mesh, take a snapshot with the wall shear stress, read a mesh file.

    listed()             the cases
    draw(rng)            one more of the same ranges
    prepare(case, seed)  what the program has in hand before the call
    run(state)           one pass, and its outputs
    work(case)           bytes and operations a pass cannot do without
    exact(case, seed)    the floating outputs in 64 bits, from plain torch

The meshes are the seeded generators' (pv2013_gb300.cases); a case fixes the
mesh (and so the work), the seed the flow through it: inlet speed and period,
relaxation time, outlet density; the mesh cases take the facets in another
order and move the grid, or the mesh, a little.
"""
import dataclasses
import functools
import math
import os
import tempfile

import numpy as np
import torch

from pv2013_gb300 import BoundarySpec, Geometry, Reader, Simulation, _capi, cases as synth
from pv2013_gb300.engine import Snapshot

STORE_BYTES = {"f64": 8, "f32": 4, "f16s": 2, "bf16s": 2}


def listed():
    return [
        # The production workload: the depth-5 vascular tree (10 million fluid nodes), 16-bit storage,
        # half a pulsation period between two field snapshots that go to pinned buffers.  The largest.
        {"name": "tree_f16s_aa", "what": "run", "shape": "tree", "depth": 5, "Q": 19, "precision": "f16s",
         "pattern": "aa", "steps": 500, "graph": True, "pinned": True},
        # The middle of the range: a bifurcation (1 million nodes) in FP32 on two lattices.
        {"name": "bifurcation_f32_pull", "what": "run", "shape": "bifurcation", "scale": 1.0, "Q": 19,
         "precision": "f32", "pattern": "pull", "steps": 250, "graph": True, "pinned": True},
        # The same vessel with the larger velocity set and 16-bit storage, in place.
        {"name": "bifurcation_d3q27_f16s", "what": "run", "shape": "bifurcation", "scale": 1.0, "Q": 27,
         "precision": "f16s", "pattern": "aa", "steps": 250, "graph": True, "pinned": True},
        # Parameter study: 24 vessels of different sizes, relaxation times and pulses in one simulation.
        {"name": "ensemble24_f16s_aa", "what": "run", "shape": "ensemble", "count": 24, "Q": 19, "precision": "f16s",
         "pattern": "aa", "steps": 200, "graph": True, "pinned": True},
        # The reference's arithmetic: FP64, the constructor's defaults, on the straight pipe (150 thousand nodes).
        {"name": "pipe_f64_pull", "what": "run", "shape": "pipe", "radius": 20, "length": 120, "Q": 19,
         "precision": "f64", "pattern": "pull", "steps": 100, "graph": False, "pinned": False},
        # The same arithmetic on a vessel of everyday size, in place, replayed as a graph.
        {"name": "vessel_f64_aa", "what": "run", "shape": "vessel", "vessel": 4003, "Q": 19, "precision": "f64",
         "pattern": "aa", "steps": 101, "graph": True, "pinned": False},
        # A small, ragged vessel in BF16 with an odd step count and no graph: launches and gaps.
        {"name": "vessel_bf16s_odd", "what": "run", "shape": "vessel", "vessel": 4005, "Q": 19, "precision": "bf16s",
         "pattern": "aa", "steps": 77, "graph": False, "pinned": False},
        # The smallest call: a few steps of a short pipe and its monitors (a convergence loop's body).
        {"name": "pipe_f32_monitors", "what": "monitor", "shape": "pipe", "radius": 9, "length": 40, "Q": 19,
         "precision": "f32", "pattern": "aa", "steps": 10, "graph": False, "pinned": False},
        # Starting the production run: voxelize and classify the tree's mesh, build the lattice, and the
        # monitors after the first steps.
        {"name": "setup_tree_f16s", "what": "setup", "shape": "tree", "depth": 5, "Q": 19, "precision": "f16s",
         "pattern": "aa", "steps": 20},
        # Meshing a bifurcation on a finer grid: node types and boundary lists alone.
        {"name": "voxelize_bifurcation", "what": "voxelize", "shape": "bifurcation", "scale": 1.0, "spacing": 0.75},
        # A snapshot of the running flow with the wall shear stress.
        {"name": "snapshot_bifurcation", "what": "snapshot", "shape": "bifurcation", "scale": 1.0, "Q": 19,
         "precision": "f32", "pattern": "aa", "steps": 2, "graph": False},
        # Reading a vessel's ASCII STL file.
        {"name": "stl_ascii_vessel", "what": "stl", "shape": "vessel", "vessel": 4001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any storage, pattern, velocity set and launch mode on a vessel, pipe, bifurcation or ensemble
    of any size below the tree's, or another set-up, snapshot or file of the listed kinds."""
    what = rng.choice(["run"] * 6 + ["monitor", "setup", "voxelize", "snapshot", "stl"])
    shape = rng.choice(["pipe", "vessel", "bifurcation", "ensemble"] if what == "run" else ["pipe", "vessel", "bifurcation"])
    case = {"what": what, "shape": shape}
    if shape == "pipe":
        case["radius"] = _log_int(rng, 6, 40)
        case["length"] = _log_int(rng, max(20, 2 * case["radius"]), 400)
    elif shape == "vessel":
        case["vessel"] = rng.randrange(4000, 4064)
    elif shape == "bifurcation":
        case["scale"] = round(rng.uniform(0.5, 1.2), 3)
    else:
        case["count"] = rng.randrange(2, 17)
        case["first"] = rng.randrange(4000, 4064)
    if what == "voxelize":
        case["spacing"] = round(rng.uniform(0.7, 1.6), 3)
    if what in ("voxelize", "stl"):
        return case
    case["Q"] = rng.choice([19, 19, 19, 27])
    case["precision"] = rng.choice(["f16s", "f16s", "f32", "bf16s", "f64"])
    case["pattern"] = rng.choice(["aa", "aa", "pull"])
    big = case["precision"] == "f64" or shape == "ensemble"
    case["steps"] = _log_int(rng, 1, 40) if what != "run" else _log_int(rng, 20, 150 if big else 400)
    if what != "setup":
        case["graph"] = rng.random() < 0.6
        case["corrections"] = rng.choice([0, 0, 0, 1, 2, 3])
    if what == "run":
        case["pinned"] = rng.random() < 0.5
    return case


# ---------------------------------------------------------------------------------------------------------------------
# inputs

@functools.lru_cache(maxsize=4)
def _tree(depth):
    return synth.vascular_tree(depth=depth)


@functools.lru_cache(maxsize=80)
def _vessel(k):
    return synth.vessel(k)


@functools.lru_cache(maxsize=8)
def _bifurcation(scale):
    n = [int(round(v * scale)) for v in (256, 512, 256)]
    return synth.bifurcation(n[0], n[1], n[2], r_parent=24.0 * scale, r_child=18.0 * scale)


@functools.lru_cache(maxsize=16)
def _pipe(radius, length):
    side = 2 * (radius + 4)
    return synth.pipe(radius=float(radius), length=float(length), ny=length + 8, nxz=side)


def _meshes(case):
    """The case's vessels (one, or an ensemble's)."""
    s = case["shape"]
    if s == "tree":
        return [_tree(case["depth"])]
    if s == "vessel":
        return [_vessel(case["vessel"])]
    if s == "bifurcation":
        return [_bifurcation(case["scale"])]
    if s == "pipe":
        return [_pipe(case["radius"], case["length"])]
    return [_vessel(4000 + (case.get("first", 4000) - 4000 + i) % 64) for i in range(case["count"])]


class _Flow:
    """The flow a seed draws through one vessel."""

    def __init__(self, mesh, rng):
        self.mesh = mesh
        self.tau = float(rng.uniform(0.75, 1.0))
        self.u_max = float(rng.uniform(0.02, 0.04))
        self.rho_out = float(rng.uniform(0.998, 1.002))
        period = int(rng.integers(500, 1500))
        phase = float(rng.uniform(0.0, 2.0 * math.pi))
        t = np.arange(period, dtype=np.float64)
        self.amp = self.u_max * (1.0 + 0.5 * np.sin(2.0 * np.pi * t / period + phase))

    def specs(self, geom, Q):
        profile = self.mesh.inlet_profile(geom)
        if Q == 19:
            return [BoundarySpec(synth.INLET_LIST, _capi.BC_VEL_NEGY, dir=(0.0, -1.0, 0.0), profile=profile, amp=self.amp),
                    BoundarySpec(synth.OUTLET_LIST, _capi.BC_PRESS_POSY, rho=self.rho_out)]
        return [BoundarySpec(synth.INLET_LIST, _capi.BC_VELOCITY, dir=(0.0, -1.0, 0.0), profile=profile, amp=self.amp,
                             face=_capi.FACE_NEGY),
                BoundarySpec(synth.OUTLET_LIST, _capi.BC_PRESSURE, rho=self.rho_out, face=_capi.FACE_POSY)]


def _flows(case, seed):
    rng = np.random.default_rng(seed)
    return [_Flow(m, rng) for m in _meshes(case)]


def _simulation(case, flows, geoms):
    opts = dict(Q=case["Q"], precision=case["precision"], pattern=case["pattern"], corrections=case.get("corrections", 0))
    specs = [f.specs(g, case["Q"]) for f, g in zip(flows, geoms)]
    if case["shape"] == "ensemble":
        return Simulation(geoms, [f.tau for f in flows], specs, **opts)
    return Simulation(geoms[0], flows[0].tau, specs[0], **opts)


def _moved(mesh, seed):
    """The mesh moved and scaled by less than a part in ten thousand (another scan of the same vessel)."""
    rng = np.random.default_rng(seed)
    t = mesh.triangles.copy()
    t[:, :9] = t[:, :9] * (1.0 + 1e-5 * rng.random()) + np.tile(1e-4 * rng.random(3), 3)
    return t


def _turned(mesh, seed):
    """The same surface written in another order: the facets from a seeded one on, then those before it."""
    return np.roll(mesh.triangles, int(np.random.default_rng(seed).integers(len(mesh.triangles))), axis=0)


def _window(mesh, spacing, seed):
    """A grid of the given spacing around the mesh, with a seeded margin of 1 to 5 points before it; a bit over a third
    of a spacing off, so that no grid plane lies on the mesh's flat ends."""
    v = mesh.triangles[:, :9].reshape(-1, 3)
    lo, hi = v.min(axis=0), v.max(axis=0)
    before = np.random.default_rng(seed).integers(1, 6, 3)
    return (tuple(float(a) - (int(k) + 0.37) * spacing for a, k in zip(lo, before)),
            tuple(int(math.ceil(d / spacing)) + 8 for d in hi - lo))


class _File:
    """A file that goes with its last user."""

    def __init__(self, triangles):
        fd, self.path = tempfile.mkstemp(suffix=".stl")
        os.close(fd)
        Reader.writeSTLASCII(self.path, triangles)

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def prepare(case, seed):
    what = case["what"]
    if what == "stl":
        return {"what": what, "file": _File(_moved(_meshes(case)[0], seed))}
    if what == "voxelize":
        m = _meshes(case)[0]
        return {"what": what, "triangles": _turned(m, seed), "spacing": case["spacing"],
                "grid": _window(m, case["spacing"], seed),
                "predicates": [dataclasses.replace(p, tol=case["spacing"]) for p in m.predicates]}
    flows = _flows(case, seed)
    if what == "setup":
        m = flows[0].mesh
        t = torch.empty((len(m.triangles), 12), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        np.copyto(t, _turned(m, seed))
        return {"what": what, "case": dict(case), "flows": flows, "triangles": t}
    geoms = [f.mesh.geometry() for f in flows]
    sim = _simulation(case, flows, geoms)
    if what == "monitor":
        sim.set_divergence_tolerance(0.5)       # an open vessel fills by a few percent while the flow starts
    state = {"what": what, "sim": sim, "steps": case["steps"], "graph": case["graph"], "out": None}
    if what == "snapshot":
        state["snapshot"] = Snapshot(sim)
    elif case.get("pinned"):
        n = sim.info().n_nodes
        pin = torch.cuda.is_available()
        state["out"] = (None, torch.empty(n, dtype=torch.float64, pin_memory=pin).numpy(),
                        torch.empty((n, 3), dtype=torch.float64, pin_memory=pin).numpy())
    return state


def run(state):
    what = state["what"]
    if what == "run":
        sim = state["sim"]
        sim.step(state["steps"], graph=state["graph"])
        _, rho, u = sim.fields(f=False, out=state["out"])
        return {"rho": rho, "u": u}
    if what == "monitor":
        sim = state["sim"]
        sim.step(state["steps"], graph=state["graph"], monitor=True)
        return sim.monitors()
    if what == "snapshot":
        sim, snap = state["sim"], state["snapshot"]
        sim.step(state["steps"], graph=state["graph"])
        snap.capture()
        rho, u, wss, _ = snap.data()
        return {"rho": rho, "u": u, "wss": wss}
    if what == "stl":
        tris, _ = Reader.readSTLASCIIDevice(state["file"].path)
        return tris
    if what == "voxelize":
        geom = Geometry(state["triangles"], state["spacing"], grid=state["grid"], predicates=state["predicates"])
        return {"flags": geom.flags(), "boundary": geom.boundaryPoints, "wall": geom.WallboundaryPoints}
    case, flow = state["case"], state["flows"][0]
    mesh = flow.mesh
    geom = Geometry(state["triangles"], mesh.spacing, grid=mesh.grid, predicates=mesh.predicates)
    sim = _simulation(case, [flow], [geom])
    sim.step(case["steps"])
    return {"nodes": sim.nodes(), "boundary": geom.boundaryPoints, "inlet": geom.InletboundaryPoints,
            "monitors": sim.monitors()}


@functools.lru_cache(maxsize=64)
def _counts(key):
    """(fluid nodes, boundary points, grid points, triangles) of a case."""
    case = dict(key)
    nf = nb = npts = nt = 0
    for m in _meshes(case):
        g = Geometry(m.triangles, case["spacing"], grid=_window(m, case["spacing"], 0)) if "spacing" in case else m.geometry()
        nf += int(g.info.n_fluid)
        nb += int(g.info.n_boundary)
        npts += int(g.info.n_points)
        nt += len(m.triangles)
    return nf, nb, npts, nt


def work(case):
    """Of the iterations: each step's populations read and written once (the method's 2 Q values per node update),
    then rho and u written.  Of the meshing: the triangles read, one byte per grid point and the lists written."""
    nf, nb, npts, nt = _counts(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    what = case["what"]
    if what == "stl":
        return {"bytes": 96 * nt + 280 * nt, "flops": 12 * 20 * nt}
    if what == "voxelize":
        return {"bytes": 96 * nt + npts + 16 * nb, "flops": 60 * nt}
    Q = case["Q"]
    s = STORE_BYTES[case["precision"]]
    if what == "setup":
        return {"bytes": 96 * nt + npts + 16 * nb + nf * (Q * s + 8) + 2 * Q * s * nf * case["steps"],
                "flops": 60 * nt + (200 if Q == 19 else 290) * nf * case["steps"]}
    update = 200 if Q == 19 else 290
    bytes_ = 2 * Q * s * nf * case["steps"]
    flops = update * nf * case["steps"]
    if what == "run":
        bytes_ += nf * (Q * s + 32)
    elif what == "monitor":
        bytes_ += nf * Q * s
    else:
        bytes_ += nf * (Q * s + 32) + 8 * nb
    return {"bytes": bytes_, "flops": flops + 60 * nf}


# ---------------------------------------------------------------------------------------------------------------------
# the same results in 64 bits, from plain torch

def _lattice(Q):
    if Q == 19:
        c = [[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [1, -1, 0], [1, 0, 1], [1, 0, -1],
             [-1, 1, 0], [-1, -1, 0], [-1, 0, 1], [-1, 0, -1], [0, 1, 1], [0, 1, -1], [0, -1, 1], [0, -1, -1], [0, 0, 0]]
        w = [2 / 36] * 6 + [1 / 36] * 12 + [12 / 36]
    else:
        c = [[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [1, -1, 0], [-1, 1, 0],
             [-1, -1, 0], [1, 0, 1], [-1, 0, 1], [1, 0, -1], [-1, 0, -1], [0, 1, 1], [0, 1, -1], [0, -1, 1], [0, -1, -1],
             [1, 1, 1], [-1, -1, -1], [1, 1, -1], [-1, -1, 1], [1, -1, 1], [-1, 1, -1], [1, -1, -1], [-1, 1, 1]]
        w = [8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8
    return c, w, [c.index([-a for a in v]) for v in c]


def _flags(mesh, dev):
    """Fluid points of the mesh's grid: an odd number of surface crossings above the point."""
    mn, dims = mesh.grid
    Nx, Ny, Nz = (int(v) for v in dims)
    T = torch.from_numpy(np.ascontiguousarray(mesh.triangles)).to(dev).reshape(-1, 4, 3)
    T, normal = T[:, :3] - torch.tensor([float(v) for v in mn], dtype=torch.float64, device=dev), T[:, 3]
    hist = torch.zeros((Nx * Ny, Nz + 1), dtype=torch.int8, device=dev)
    lo = torch.ceil(T[:, :, :2].amin(1))
    span = (torch.floor(T[:, :, :2].amax(1)) - lo).amax(0).long().tolist()
    (x1, y1, z1), (x2, y2, _), (x3, y3, _) = [T[:, k].unbind(1) for k in range(3)]
    for di in range(span[0] + 1):
        for dj in range(span[1] + 1):
            x, y = lo[:, 0] + di, lo[:, 1] + dj
            a = (x2 - x) * (y3 - y) - (x3 - x) * (y2 - y)
            b = (x3 - x) * (y1 - y) - (x1 - x) * (y3 - y)
            c = (x1 - x) * (y2 - y) - (x2 - x) * (y1 - y)
            hit = (normal[:, 2] != 0) & (((a >= 0) & (b >= 0) & (c >= 0)) | ((a <= 0) & (b <= 0) & (c <= 0)))
            hit &= (x >= 0) & (x < Nx) & (y >= 0) & (y < Ny)
            z = z1 + ((x1 - x) * normal[:, 0] + (y1 - y) * normal[:, 1]) / normal[:, 2]   # on the facet's plane
            k = hit.nonzero().squeeze(1)
            z = z + 1e-7 * (Nz - 1 + 0.1)                             # the ray test's tolerance at its start
            top = torch.floor(z[k]).clamp(-1, Nz - 1).long() + 1      # the points below the crossing: 0 .. top-1
            col = (x[k] * Ny + y[k]).long()
            hist.view(-1).index_add_(0, col * (Nz + 1) + top, torch.ones_like(top, dtype=torch.int8))
    odd = hist.flip(1).cumsum(1, dtype=torch.int32).flip(1)[:, 1:] & 1
    return odd.bool().reshape(Nx, Ny, Nz)


def _grow(m):
    """Points with a True point among their 26 neighbours or themselves."""
    for ax in range(3):
        n = m.shape[ax]
        o = m.clone()
        o.narrow(ax, 1, n - 1).logical_or_(m.narrow(ax, 0, n - 1))
        o.narrow(ax, 0, n - 1).logical_or_(m.narrow(ax, 1, n - 1))
        m = o
    return m


class _Exact:
    """One vessel's flow in 64 bits: BGK, bounce-back walls, Zou-He velocity inlet and pressure outlets."""

    def __init__(self, flow, Q, corrections, dev):
        self.flow, self.Q, self.dev = flow, Q, dev
        self.c, self.w, self.opp = _lattice(Q)
        self.all_dirs, self.fix_lists = bool(corrections & 1), bool(corrections & 2)
        mesh = flow.mesh
        fluid = _flags(mesh, dev)
        pad = torch.zeros([n + 2 for n in fluid.shape], dtype=torch.bool, device=dev)
        pad[1:-1, 1:-1, 1:-1] = fluid
        bound = (_grow(~pad) & pad)[1:-1, 1:-1, 1:-1]
        pts = fluid.reshape(-1).nonzero().squeeze(1)
        self.N = len(pts)
        b = bound.reshape(-1)[pts]
        dims = [int(v) for v in mesh.grid[1]]
        ijk = torch.stack([pts // (dims[1] * dims[2]), (pts // dims[2]) % dims[1], pts % dims[2]], 1)
        xyz = ijk.double() + torch.tensor([float(v) for v in mesh.grid[0]], dtype=torch.float64, device=dev)
        role = torch.where(b, 1, 0)
        for p in reversed(sorted(mesh.predicates, key=lambda p: p.list_id)):
            m = b & ((xyz[:, p.axis] - float(p.plane)).abs() <= p.tol)
            for a in range(3):
                if a != p.axis:
                    m &= (xyz[:, a] > p.lo[a]) & (xyz[:, a] < p.hi[a])
            role[m] = 2 + p.list_id
        self.role = role
        self.inlet = (role == 2 + synth.INLET_LIST).nonzero().squeeze(1)
        self.outlet = (role == 2 + synth.OUTLET_LIST).nonzero().squeeze(1)
        cx, cz = mesh.inlet.center
        r2 = (xyz[self.inlet, 0] - cx) ** 2 + (xyz[self.inlet, 2] - cz) ** 2
        self.profile = (1.0 - r2 / mesh.inlet.radius ** 2).clamp(min=0.0)
        number = torch.full([n + 2 for n in fluid.shape], -1, dtype=torch.int32, device=dev)
        number[1:-1, 1:-1, 1:-1].masked_scatter_(fluid, torch.arange(self.N, dtype=torch.int32, device=dev))
        self.dims = [n + 2 for n in fluid.shape]
        self.flat = ((ijk[:, 0] + 1) * self.dims[1] + ijk[:, 1] + 1) * self.dims[2] + ijk[:, 2] + 1
        self.number = number.reshape(-1)
        del fluid, pad, bound
        self.src, self.missing = [], []
        for v in self.c:
            s = self.number[self.flat - self._shift(v)].long()
            self.missing.append((s < 0).nonzero().squeeze(1))
            self.src.append(torch.where(s < 0, 0, s).to(torch.int32))
        self.f = torch.tensor(self.w, dtype=torch.float64, device=dev)[:, None].repeat(1, self.N)
        self.step_no = 0

    def _shift(self, v):
        return (v[0] * self.dims[1] + v[1]) * self.dims[2] + v[2]

    def _sums(self, f):
        rho = f.sum(0)
        m = [torch.zeros_like(rho) for _ in range(3)]
        for q, v in enumerate(self.c):
            for a in range(3):
                if v[a]:
                    m[a].add_(f[q], alpha=v[a])
        return rho, [x / rho for x in m]

    def macro(self):
        rho, u = self._sums(self.f)
        return rho, torch.stack(u, 1)

    def step(self):
        om = 1.0 / self.flow.tau
        f = self.f
        rho, u = self._sums(f)
        base = 1.0 - 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        post = torch.empty_like(f)
        for q, v in enumerate(self.c):
            du = sum((u[a] * float(v[a]) for a in range(3) if v[a]), torch.zeros_like(rho))
            post[q] = f[q] + om * (self.w[q] * rho * (base + du * (3.0 + 4.5 * du)) - f[q])
        never = self.opp[0] if self.Q == 19 and not self.all_dirs else -1
        for q in range(self.Q):
            torch.index_select(post[q], 0, self.src[q], out=f[q])
            m = self.missing[q]
            bounced = torch.full_like(f[q][m], self.w[q])
            if q != never:
                wall = (self.role[m] == 1) | self.fix_lists
                bounced = torch.where(wall, post[self.opp[q]][m], bounced)
            f[q][m] = bounced
        amp = self.flow.amp[self.step_no % len(self.flow.amp)]
        self._face(self.inlet, -1, speed=-amp * self.profile)
        self._face(self.outlet, 1, density=self.flow.rho_out)
        self.step_no += 1

    def _face(self, nodes, sg, speed=None, density=None):
        """Zou-He on nodes whose unknown populations have c_y = sg."""
        if not len(nodes):
            return
        c, p = self.c, self.f[:, nodes]
        known = sum(p[q] for q in range(self.Q) if c[q][1] == 0) + 2.0 * sum(p[q] for q in range(self.Q) if c[q][1] == -sg)
        if speed is not None:
            uy, rho = speed, known / (1.0 - sg * speed)
        else:
            uy, rho = sg * (1.0 - known / density), density
        ka = 0.5 if self.Q == 19 else 1.0 / 6.0
        N = [ka * sum(p[q] * c[q][a] for q in range(self.Q) if c[q][1] == 0 and c[q][a]) for a in (0, 2)]
        for q in range(self.Q):
            if c[q][1] == sg:
                self.f[q, nodes] = p[self.opp[q]] + 6.0 * self.w[q] * rho * sg * uy - c[q][0] * N[0] - c[q][2] * N[1]

    def wss(self, u):
        """|mu g| at the wall nodes, g the mean velocity difference to the neighbours that are fluid points."""
        wall = (self.role == 1).nonzero().squeeze(1)
        g, n = torch.zeros((len(wall), 3), dtype=torch.float64, device=self.dev), torch.zeros(len(wall), device=self.dev)
        for v in self.c:
            s = self.number[self.flat[wall] + self._shift(v)].long()
            ok = s >= 0
            g += torch.where(ok[:, None], u[s.clamp(min=0)] - u[wall], 0.0)
            n += ok
        return ((2.0 * self.flow.tau - 1.0) / 6.0) * (g / n[:, None]).norm(dim=1)


def exact(case, seed):
    what = case["what"]
    if what == "voxelize":
        return None                     # node types and lists are whole numbers
    if what == "stl":
        return _moved(_meshes(case)[0], seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    parts = []
    for flow in _flows(case, seed):
        e = _Exact(flow, case["Q"], case.get("corrections", 0), dev)
        for _ in range(case["steps"]):
            e.step()
        rho, u = e.macro()
        if what in ("monitor", "setup"):
            sp = u.norm(dim=1)
            m = {"step": case["steps"], "mass": float(rho.sum()), "inlet_flux": float((rho * sp)[e.inlet].sum()),
                    "outlet_flux": float((rho * sp)[e.outlet].sum()), "max_speed": float(sp.max()), "nonfinite": False}
            return m if what == "monitor" else {"nodes": None, "boundary": None, "inlet": None, "monitors": m}
        parts.append((rho, u, e.wss(u) if what == "snapshot" else None))
        del e
    out = {"rho": torch.cat([p[0] for p in parts]), "u": torch.cat([p[1] for p in parts])}
    if what == "snapshot":
        out["wss"] = parts[0][2]
    return out
