"""Timed workloads of the coupled immersed-boundary lattice-Boltzmann step, through the public API.

``listed()`` gives the workloads, ``draw(rng)`` one more of the same ranges, ``prepare(case, seed)`` the
objects a driver program holds (context, lattice, particles, page-locked result arrays), ``run(state)``
one output interval of such a driver: some time steps, then the results it writes.  ``work(case)`` counts
what an interval cannot do without and ``exact(case, seed)`` is the same interval in plain 64-bit torch.

Results come in the precision the lattice is stored in: a driver keeps the velocity field and the
particle data of an FP32 or FP16 run in 32 or 16 bits for its analysis on the GPU.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import biblbm_gb300 as bib
from biblbm_gb300 import meshes

BYTES = {"f64": 8, "f32": 4, "f16": 2}
TORCH = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16}
BODY, U_WALL, U_TGV, TAU = 1e-6, 0.01, 0.02, 1.0
PIPE_PP = (1.0, 1.5, 1e-5)  # Morse potential between cells: range, beta, strength
PIPE_WALL = (2.0, 1e-5)     # spring potential of the pipe's wall: range, strength
BATCH_EDGES = (32, 48, 64, 80, 96)


def coupled(name, nx, ny, nz, walls, storage, shape, radius, cells, level, steps, dirac="roma", spread="atomic", lam=1.0, read="end"):
    c = dict(kind="coupled", nx=nx, ny=ny, nz=nz, walls=walls, storage=storage, shape=shape, radius=radius, cells=cells, level=level,
             steps=steps, dirac=dirac, spread=spread, lam=lam, read=read)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the dense red-cell suspension in a channel, the benchmark's default: 20 % haematocrit, FP16
        coupled("channel_f16", 512, 128, 128, "channel", "f16", "rbc", 13.9, 400, 3, 50),
        # a suspension with the smoother 4-point kernel, in FP32, on rows that are no power of two
        coupled("channel_peskin_f32", 240, 96, 90, "channel", "f32", "rbc", 10.0, 200, 3, 50, dirac="peskin"),
        # a long thin channel whose rows exceed a tile of the staged kernel, reproducible spreading
        coupled("channel_long_det_f16", 1024, 64, 64, "channel", "f16", "rbc", 10.0, 260, 3, 50, spread="deterministic"),
        # one finely meshed red cell in simple shear, the FP32 run of a single-cell study
        coupled("rbc_shear_f32", 128, 64, 64, "shear", "f32", "rbc", 8.0, 1, 4, 100),
        # one capsule in simple shear in the reference's own arithmetic
        coupled("capsule_f64", 64, 64, 64, "shear", "f64", "capsule", 10.0, 1, 3, 50),
        # the smallest: a coarse capsule on N + 1 = 33 nodes, every step's cell data read by the driver
        coupled("capsule_small_read_f32", 33, 33, 33, "shear", "f32", "capsule", 5.5, 1, 2, 20, read="step"),
        # a capsule whose interior is five times as viscous: the phase field follows the membrane
        coupled("capsule_lambda_f32", 80, 80, 80, "shear", "f32", "capsule", 13.0, 1, 3, 100, lam=5.0),
        # red cells in a pipe with pair repulsion and a repulsive wall
        coupled("pipe_f32", 192, 50, 50, "pipe", "f32", "rbc", 7.5, 40, 3, 50),
        # a parameter study: independent capsules of uneven sizes stepped as one batch
        dict(name="batch_f32", kind="batch", storage="f32", count=64, mix=4, steps=20),
        # the lattice alone: two-relaxation-time Taylor-Green flow, the largest box of the sweep
        dict(name="lattice_trt_f16", kind="lattice", nx=384, ny=384, nz=384, collision="trt", storage="f16", steps=60),
        # the lattice alone on N + 1 nodes (odd rows)
        dict(name="lattice_odd_f32", kind="lattice", nx=201, ny=201, nz=201, collision="bgk", storage="f32", steps=20),
        # the reference's co-processor offload: populations sent, collided and received in its wire order
        dict(name="coprocessor_f64", kind="coprocessor", nx=128, ny=96, nz=80, storage="f64", steps=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _level(rng, radius):
    """A mesh refinement whose edges are 0.35 to 2.6 lattice units long."""
    return rng.choice([m for m in (2, 3, 4) if 0.35 <= 1.1 * radius / 2 ** m <= 2.6] or [4])


def draw(rng):
    kind = rng.choice(["channel", "channel", "shear", "shear", "pipe", "batch", "lattice", "lattice", "coprocessor"])
    storage = rng.choice(["f16", "f32", "f32", "f64"])
    if kind == "batch":
        return dict(kind="batch", storage=rng.choice(["f32", "f16"]), count=_log(rng, 2, 64), mix=rng.randrange(1 << 20), steps=rng.randrange(10, 21))
    if kind == "lattice":
        top = 320 if storage != "f64" else 128
        nx, ny, nz = (_log(rng, 24, top) for _ in range(3))
        return dict(kind="lattice", nx=nx, ny=ny, nz=nz, collision=rng.choice(["trt", "bgk", "bgk_guo_vof"]), storage=storage, steps=rng.randrange(10, 41))
    if kind == "coprocessor":
        return dict(kind="coprocessor", nx=_log(rng, 16, 160), ny=_log(rng, 16, 100), nz=_log(rng, 16, 100), storage=storage, steps=rng.randrange(1, 4))
    dirac, spread = rng.choice(["roma", "roma", "peskin"]), rng.choice(["atomic", "atomic", "deterministic"])
    steps = rng.randrange(20, 61)
    if kind == "shear":
        top = 128 if storage != "f64" else 64
        nx, ny, nz = _log(rng, 30, 2 * top), _log(rng, 30, top), _log(rng, 30, top)
        radius = round(min(nx, ny, nz) / rng.uniform(4.0, 7.0), 2)
        return coupled(None, nx, ny, nz, "shear", storage, rng.choice(["capsule", "rbc"]), radius, 1, _level(rng, radius), steps, dirac, spread,
                       rng.choice([1.0, 1.0, 5.0]), rng.choice(["end", "end", "step"]))
    radius = round(rng.uniform(6.0, 14.0), 2)
    side = int(radius * rng.uniform(4.5, 8.0))
    nx = _log(rng, 5 * radius, 1200 if storage != "f64" else 160)
    if kind == "pipe":
        return coupled(None, nx, side + 6, side + 6, "pipe", storage, "rbc", radius, _log(rng, 2, 80), 3, steps, dirac, spread)
    return coupled(None, nx, side, int(side * rng.uniform(0.8, 1.2)), "channel", storage, "rbc", radius, _log(rng, 4, 300), 3, steps, dirac,
                   spread)


# ---------------------------------------------------------------- the physical set-up
_MESH = {}


def _mesh(shape, level, radius):
    if (shape, level) not in _MESH:
        xyz, tri = meshes.evans_fung(level, 1.0) if shape == "rbc" else meshes.icosphere(level, 1.0)
        _MESH[shape, level] = (xyz - xyz.mean(axis=0), tri)
    xyz, tri = _MESH[shape, level]
    return xyz * radius, tri


def _area_volume(xyz, tri):
    a, b, c = xyz[tri[:, 0]], xyz[tri[:, 1]], xyz[tri[:, 2]]
    n = np.cross(b - a, c - a)
    return 0.5 * np.linalg.norm(n, axis=1).sum(), np.einsum("ij,ij->i", a, np.cross(b, c)).sum() / 6.0


def _sites(case):
    """Centres of a regular arrangement of the cells that keeps them apart: disc-like cells lie flat."""
    r, n = case["radius"], (case["nx"], case["ny"], case["nz"])
    if case["cells"] == 1:
        return np.array([[0.5 * (m - 1) for m in n]])
    pitch = (2 * r + 1, 2 * r + 1, 2 * (0.34 + math.sin(0.28)) * r + 1)
    axes = []
    for a in range(3):
        lo, hi = (0.0, n[a]) if a == 0 else (1.5, n[a] - 2.5)
        m = max(1, int((hi - lo) / pitch[a]))
        axes.append(lo + (np.arange(m) + 0.5) * (hi - lo) / m)
    s = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    if case["walls"] == "pipe":
        y0, z0, pr = _pipe(case)
        d = np.hypot(s[:, 1] - y0, s[:, 2] - z0)
        s = s[d <= max(d.min() + 1e-9, pr - r - 1.6)]
    return s


def _pipe(case):
    return 0.5 * (case["ny"] - 1), 0.5 * (case["nz"] - 1), 0.5 * (min(case["ny"], case["nz"]) - 5)


def _n_cells(case):
    return min(case["cells"], len(_sites(case)))


def _setup(case, seed):
    """Everything the run is made of, as numpy: lattice arguments, initial velocity, mesh, parameters, positions."""
    rng = np.random.default_rng(seed)
    nx, ny, nz, r = case["nx"], case["ny"], case["nz"], case["radius"]
    rest, tri = _mesh(case["shape"], case["level"], r)
    area, vol = _area_volume(rest, tri)
    nu = (TAU - 0.5) / 3
    shear = case["walls"] == "shear"
    rate = 2 * U_WALL / (ny - 1) if shear else BODY * ny / (2 * nu)
    G = nu * rate * r / 0.1  # capillary number 0.1
    if case["shape"] == "capsule":
        model, prm = "capsule_skalak", bib.membrane_params(G=G, C=1.0)
    else:
        model = "skalak_bending"
        prm = bib.membrane_params(G=G, C=1.0, k_area_global=1.0, k_volume=1.0, vol_desired=vol, k_bend=0.01 * G * area)
    sites = _sites(case)
    sites = sites[rng.permutation(len(sites))[: case["cells"]]] + rng.uniform(-0.3, 0.3, (min(len(sites), case["cells"]), 3))
    pos = []
    for s in sites:
        if len(sites) == 1:
            q = meshes.random_rotation(rng)
        else:  # tilted out of the flow-vorticity plane by up to 0.28, turned freely about its axis
            q = meshes.rotation_matrix((math.cos(t := rng.uniform(0, 2 * math.pi)), math.sin(t), 0), rng.uniform(0, 0.28))
            q = q @ meshes.rotation_matrix((0, 0, 1), rng.uniform(0, 2 * math.pi))
        pos.append(rest @ q.T + s)
    lattice = dict(collision="bgk_guo_vof", omega=1 / TAU, storage=case["storage"])
    y, z = np.arange(ny), np.arange(nz)
    u = np.zeros((3, nz, ny, nx))
    if shear:
        lattice.update(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=[[-U_WALL, 0, 0], [U_WALL, 0, 0], [0, 0, 0], [0, 0, 0]])
        u[0] = (U_WALL * (2 * y / (ny - 1) - 1))[None, :, None]
    elif case["walls"] == "channel":
        lattice.update(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb", body_force=(BODY, 0, 0))
        top = BODY * min(ny, nz) ** 2 / (8 * nu)
        u[0] = (top * (1 - ((2 * y + 1) / ny - 1) ** 2)[None, :] * (1 - ((2 * z + 1) / nz - 1) ** 2)[:, None])[:, :, None]
    else:
        lattice.update(periodic=(1, 1, 1), body_force=(BODY, 0, 0))
        y0, z0, pr = _pipe(case)
        rr = (y[None, :] - y0) ** 2 + (z[:, None] - z0) ** 2
        u[0] = (BODY / (4 * nu) * np.maximum(pr * pr - rr, 0))[:, :, None]
    if case["lam"] != 1.0:
        lattice.update(use_phase=True, omega_inner=1 / (0.5 + 3 * case["lam"] * nu))
    return dict(lattice=lattice, u=u, rest=rest, tri=tri, model=model, prm=prm, pos=np.array(pos))


def _flow(case, seed, device):
    """Density and velocity of a Taylor-Green vortex with seeded phases (and a weaker one along z)."""
    rng = np.random.default_rng(seed)
    ph, amp = rng.uniform(0, 2 * math.pi, 4), U_TGV * rng.uniform(0.8, 1.0)
    x, y, z = (2 * math.pi / n * torch.arange(n, dtype=torch.float64, device=device) for n in (case["nx"], case["ny"], case["nz"]))
    X, Y, Z = x[None, None, :] + ph[0], y[None, :, None] + ph[1], z[:, None, None]
    ratio = case["ny"] / case["nx"]  # divergence-free on a box of any shape, the larger component at the amplitude
    a0, a1 = amp * min(1.0, 1 / ratio), amp * min(1.0, ratio)
    shape = (case["nz"], case["ny"], case["nx"])
    u = torch.empty((3,) + shape, dtype=torch.float64, device=device)
    u[0] = a0 * torch.sin(X) * torch.cos(Y) + 0.2 * amp * torch.sin(Z + ph[2])
    u[1] = -a1 * torch.cos(X) * torch.sin(Y)
    u[2] = 0.2 * amp * torch.sin(Y + ph[3])
    rho = 1 + 0.75 * a0 * a1 * (torch.cos(2 * X) + torch.cos(2 * Y)) + torch.zeros(shape, dtype=torch.float64, device=device)
    return rho, u


def _instances(case, seed):
    """The capsules of a batch: sizes from the case, capillary numbers and orientations from the seed."""
    mix, rng = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n, level = int(mix.choice(BATCH_EDGES)), int(mix.choice([2, 3]))
        c = coupled(None, n, n, n, "shear", case["storage"], "capsule", n / 6.0, 1, level, case["steps"])
        w = _setup(c, int(rng.integers(1 << 30)))
        w["prm"] = w["prm"] * 0.1 / math.exp(rng.uniform(math.log(0.01), math.log(1.0)))
        w["prm"][1] = 1.0
        out.append((c, w))
    return out


# ---------------------------------------------------------------- the framework's side
def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _double_p(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


class _Run:
    """One lattice with its particles and the page-locked arrays its results are read into."""

    def __init__(self, ctx, case, w):
        self.ctx, self.case = ctx, case
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.lat = ctx.add_domain(nx, ny, nz, **w["lattice"])
        self.u = _pinned(3, nz, ny, nx)
        self.u.copy_(torch.from_numpy(w["u"]))
        self.lat.initialize_at_equilibrium(None, self.u.numpy())
        if case["walls"] == "pipe":
            self.lat.set_pipe_walls(*_pipe(case))
        shapes = bib.ParticleShapeLibrary(ctx)
        sid = shapes.store_mesh(w["rest"], w["tri"], "cell")
        self.fsi = bib.ImmersedBoundaryDynamics3D(self.lat, shapes, dirac=case["dirac"], spread=case["spread"])
        for p in w["pos"]:
            self.fsi.add_particle(sid, w["model"], w["prm"], p)
        if case["walls"] == "pipe":
            self.fsi.add_pp_force(bib.MorsePotential(*PIPE_PP))
            self.fsi.add_pipe_wall_interaction(bib.SpringPotential(*PIPE_WALL), *_pipe(case))
        self.fsi.init()
        self.pos = _pinned(w["pos"].shape[0] * w["pos"].shape[1], 3)
        self.stats = [_pinned(w["pos"].shape[0], 5) for _ in range(2)]

    def steps(self):
        if self.case["read"] == "end":
            self.fsi.step(self.case["steps"])
            return []
        seen = []  # the cell data of every step, waited for one step later
        for k in range(self.case["steps"]):
            self.fsi.step(1)
            self.fsi.download_async(self.stats[k % 2].numpy(), k % 2)
            if k:
                self.fsi.wait_download((k - 1) % 2)
                seen.append(self.stats[(k - 1) % 2].clone())
        self.fsi.wait_download((self.case["steps"] - 1) % 2)
        seen.append(self.stats[(self.case["steps"] - 1) % 2].clone())
        return [torch.stack(seen)]

    def results(self):
        self.fsi.download_async(self.stats[0].numpy(), 0, self.pos.numpy())
        _read_velocity(self.ctx, self.lat, self.u)
        self.fsi.wait_download(0)
        return [self.u, self.pos, self.stats[0]]


def _read_velocity(ctx, lat, u):
    ctx.check(ctx.lib.bib_lattice_get_velocity(ctx.h, lat.h, _double_p(u)))


def _kept(tensors, storage):
    """Velocity in the storage's precision, the particles' data in 32 bits at least."""
    if storage == "f64":
        return list(tensors)
    return [t.cuda().to(TORCH[storage] if k == 0 else torch.float32) for k, t in enumerate(tensors)]


def prepare(case, seed):
    ctx = bib.Context(0)
    if case["kind"] == "coupled":
        return dict(case=case, run=_Run(ctx, case, _setup(case, seed)))
    if case["kind"] == "batch":
        runs = [_Run(ctx, c, w) for c, w in _instances(case, seed)]
        return dict(case=case, ctx=ctx, runs=runs, batch=bib.Batch(ctx, [r.lat for r in runs]))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rho, u = _flow(case, seed, "cuda")
    host = _pinned(3, nz, ny, nx)
    host.copy_(u)
    tau, coll = (0.8, case["collision"]) if case["kind"] == "lattice" else (TAU, "bgk")
    lat = ctx.add_domain(nx, ny, nz, periodic=(1, 1, 1), collision=coll, omega=1 / tau, trt_magic=0.25, storage=case["storage"])
    rho_host = _pinned(nz, ny, nx)
    rho_host.copy_(rho)
    lat.initialize_at_equilibrium(rho_host.numpy(), host.numpy())
    if case["kind"] == "lattice":
        return dict(case=case, ctx=ctx, lat=lat, u=host)
    f = _pinned(nx, ny, nz, 19)
    ctx.check(ctx.lib.bib_lattice_receive(ctx.h, lat.h, f.data_ptr(), f.nbytes, 2))
    return dict(case=case, ctx=ctx, lat=lat, f=f, out=_pinned(nx, ny, nz, 19))


def run(state):
    case = state["case"]
    if case["kind"] == "coupled":
        r = state["run"]
        seen = r.steps()
        return _kept(r.results() + seen, case["storage"])
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        got = [r.results() for r in state["runs"]]
        return _kept([torch.cat([g[k].reshape(-1) for g in got]) if k else torch.cat([g[0].reshape(-1).cuda() for g in got]) for k in range(3)], case["storage"])
    ctx, lat = state["ctx"], state["lat"]
    if case["kind"] == "lattice":
        lat.collide_and_stream(case["steps"])
        _read_velocity(ctx, lat, state["u"])
        return _kept([state["u"]], case["storage"])
    f, out = state["f"], state["out"]  # CoProcessor3D: send, collideAndStream, receive
    ctx.check(ctx.lib.bib_lattice_send(ctx.h, lat.h, f.data_ptr(), f.nbytes, 2))
    lat.collide_and_stream(case["steps"])
    ctx.check(ctx.lib.bib_lattice_receive(ctx.h, lat.h, out.data_ptr(), out.nbytes, 2))
    return _kept([out], case["storage"])


def work(case):
    """Per step: the populations read and written, and for a coupled step the force read and the velocity
    written, and each vertex's position read and written; per interval the results written."""
    if case["kind"] == "batch":
        parts = [work(c) for c, _ in _instances(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, steps, s = case["nx"] * case["ny"] * case["nz"], case["steps"], BYTES[case["storage"]]
    if case["kind"] != "coupled":
        wire = (2 * 19 if case["kind"] == "coprocessor" else 3) * 8 * n
        return {"bytes": steps * 2 * 19 * s * n + wire, "flops": steps * 250 * n}
    nv = _n_cells(case) * (10 * 4 ** case["level"] + 2)
    stencil = 64 if case["dirac"] == "peskin" else 27
    field = 3 * max(s, 4) * 2
    return {"bytes": steps * (n * (2 * 19 * s + field) + nv * 48) + 24 * (n + nv),
            "flops": steps * (n * 280 + nv * (stencil * 14 + 2 * 400 + 3 * 150))}


# ---------------------------------------------------------------- the same in plain 64-bit torch
CX = (0, -1, 0, 0, -1, -1, -1, -1, 0, 0, 1, 0, 0, 1, 1, 1, 1, 0, 0)
CY = (0, 0, -1, 0, -1, 1, 0, 0, -1, -1, 0, 1, 0, 1, -1, 0, 0, 1, 1)
CZ = (0, 0, 0, -1, 0, 0, -1, 1, -1, 1, 0, 0, 1, 0, 0, 1, -1, 1, -1)
W = (1 / 3,) + tuple(1 / 18 if abs(a) + abs(b) + abs(c) == 1 else 1 / 36 for a, b, c in list(zip(CX, CY, CZ))[1:])
OPP = (0,) + tuple(range(10, 19)) + tuple(range(1, 10))
F64 = torch.float64


def _cdot(i, v):
    t = None
    for c, a in ((CX[i], v[0]), (CY[i], v[1]), (CZ[i], v[2])):
        if c:
            t = c * a if t is None else t + c * a
    return t


def _moments(f):
    rb, j = f.sum(0), []
    for c in (CX, CY, CZ):
        t = torch.zeros_like(rb)
        for i in range(19):
            if c[i]:
                t += c[i] * f[i]
        j.append(t)
    return rb, j


def _equilibrium(i, rb, j, jsq):
    if i == 0:
        return W[0] * (rb - 1.5 * jsq / (rb + 1))
    cj = _cdot(i, j)
    return W[i] * (rb + 3 * cj + (4.5 * cj * cj - 1.5 * jsq) / (rb + 1))


class _Exact:
    """f-bar = f - t_i of D3Q19 on (19, nz, ny, nx), streamed explicitly; the membranes on (cells, vertices, 3)."""

    def __init__(self, shape, omega, collision="bgk_guo_vof", walls="none", wall_u=0.0, body=0.0, omega_in=None, pipe=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.nz, self.ny, self.nx = self.shape = shape
        self.omega, self.collision, self.walls, self.wall_u, self.body, self.omega_in = omega, collision, walls, wall_u, body, omega_in
        self.F = [torch.zeros(shape, dtype=F64, device=self.dev) for _ in range(3)]
        self.per = (True, walls in ("none", "pipe"), walls != "channel")
        self.types = None
        if pipe is not None:  # 1 bounce-back outside the radius, 2 no dynamics a node further
            y, z = (torch.arange(n, dtype=F64, device=self.dev) for n in (self.ny, self.nz))
            r2 = ((y[None, :] - pipe[0]) ** 2 + (z[:, None] - pipe[1]) ** 2)[:, :, None]
            self.types = (r2 >= pipe[2] ** 2).long() + (r2 >= (pipe[2] + 1) ** 2).long()
        self.pipe, self.phase, self.X = pipe, None, None

    def start(self, rho, u):
        j = [rho * u[a] for a in range(3)]
        jsq = j[0] ** 2 + j[1] ** 2 + j[2] ** 2
        self.f = torch.stack([_equilibrium(i, rho - 1, j, jsq) for i in range(19)])
        self.fd_walls()

    def velocity(self):
        rb, j = _moments(self.f)
        u = [j[a] / (rb + 1) + 0.5 * self.F[a] for a in range(3)]
        if self.walls == "shear":
            for a in range(3):
                for y, s in ((0, -1), (self.ny - 1, 1)):
                    u[a][:, y] = s * self.wall_u if a == 0 else 0.0
        if self.types is not None:
            u = [torch.where(self.types == 0, t, torch.zeros_like(t)) for t in u]
        return torch.stack(u)

    def fd_walls(self):
        """Velocity walls at y = 0 and ny - 1: density from the known populations, stress from a one-sided difference."""
        if self.walls != "shear":
            return
        for y, o in ((0, -1), (self.ny - 1, 1)):
            uw = (o * self.wall_u, 0.0, 0.0)
            fw, f1 = self.f[:, :, y], self.f[:, :, y - o]
            on, nor = sum(fw[i] for i in range(19) if CY[i] == 0), sum(fw[i] for i in range(19) if CY[i] == o)
            vn = o * (uw[1] - 0.5 * self.F[1][:, y])
            rb = (2 * nor + on - vn) / (1 + vn)
            rb1, j1 = _moments(f1)
            du = [-o * (j1[a] / (rb1 + 1) + 0.5 * self.F[a][:, y - o] - uw[a]) for a in range(3)]
            s = -(rb + 1) / 3 / self.omega
            xy, yy, yz = du[0] * s, 2 * du[1] * s, du[2] * s
            j = [(rb + 1) * uw[a] for a in range(3)]
            jsq = j[0] ** 2 + j[1] ** 2 + j[2] ** 2
            new = [_equilibrium(i, rb, j, jsq) + 4.5 * W[i] * (2 * CX[i] * CY[i] * xy + (CY[i] ** 2 - 1 / 3) * yy + 2 * CY[i] * CZ[i] * yz) for i in range(19)]
            self.f[:, :, y] = torch.stack(new)

    def collide_and_stream(self):
        f, om = self.f, self.omega
        rb, j = _moments(f)
        out = torch.empty_like(f)
        if self.collision == "trt":
            om2, jsq = 1 / (0.25 / (1 / om - 0.5) + 0.5), j[0] ** 2 + j[1] ** 2 + j[2] ** 2
            out[0] = f[0] + om * (_equilibrium(0, rb, j, jsq) - f[0])
            for i in range(1, 10):
                e, g = _equilibrium(i, rb, j, jsq), _equilibrium(i + 9, rb, j, jsq)
                p, m = 0.5 * om * (e + g - f[i] - f[i + 9]), 0.5 * om2 * (e - g - f[i] + f[i + 9])
                out[i], out[i + 9] = f[i] + p + m, f[i + 9] + p - m
        else:
            if self.phase is not None:
                om = torch.where(self.phase, torch.full_like(rb, self.omega_in), torch.full_like(rb, om))
            forced = self.collision == "bgk_guo_vof"
            u = [j[a] / (rb + 1) + (0.5 * self.F[a] if forced else 0.0) for a in range(3)]
            J = [(rb + 1) * u[a] for a in range(3)]
            jsq = J[0] ** 2 + J[1] ** 2 + J[2] ** 2
            uF = u[0] * self.F[0] + u[1] * self.F[1] + u[2] * self.F[2]
            for i in range(19):
                out[i] = f[i] + om * (_equilibrium(i, rb, J, jsq) - f[i])
                if forced:
                    guo = -3 * uF if i == 0 else 3 * _cdot(i, self.F) - 3 * uF + 9 * _cdot(i, u) * _cdot(i, self.F)
                    out[i] += W[i] * (1 - 0.5 * om) * guo
        if self.types is not None:
            for i in range(19):
                still = torch.where(self.types == 1, f[OPP[i]], f[i])
                out[i] = torch.where(self.types == 0, out[i], still)
        for i in range(19):
            f[i] = torch.roll(out[i], (CZ[i], CY[i], CX[i]), (0, 1, 2))
            if self.walls == "channel":  # halfway bounce-back
                if CY[i]:
                    y = 0 if CY[i] > 0 else self.ny - 1
                    f[i][:, y] = out[OPP[i]][:, y]
                if CZ[i]:
                    z = 0 if CZ[i] > 0 else self.nz - 1
                    f[i][z] = out[OPP[i]][z]
        self.fd_walls()

    # ---- membranes
    def particles(self, w, dirac):
        t = lambda a, dt=F64: torch.as_tensor(a, dtype=dt, device=self.dev)  # noqa: E731
        self.X, self.tri, self.prm, self.model, self.dirac = t(w["pos"]), t(w["tri"], torch.long), [float(v) for v in w["prm"]], w["model"], dirac
        rest = t(w["rest"])
        a, b, c = (rest[self.tri[:, k]] for k in range(3))
        self.a0 = 0.5 * torch.linalg.norm(torch.cross(b - a, c - a, dim=-1), dim=-1)
        e0, e1 = b - a, c - a
        self.l0, self.l0p = torch.linalg.norm(e0, dim=-1), torch.linalg.norm(e1, dim=-1)
        self.sin0 = torch.linalg.norm(torch.cross(e0, e1, dim=-1), dim=-1) / (self.l0 * self.l0p)
        self.cos0 = (e0 * e1).sum(-1) / (self.l0 * self.l0p)
        edge, quads = {}, []  # the four vertices of each pair of triangles with a common edge
        for p, q, r in w["tri"].tolist():
            for x, y, z in ((p, q, r), (q, r, p), (r, p, q)):
                if (x, z) in edge:
                    quads.append((z, y, x, edge[x, z]))
                else:
                    edge[z, x] = y
        self.quads = t(quads, torch.long)
        _, self.c0, self.s0 = self.angles(rest[None])
        self.update()

    def angles(self, X):
        v = [X[:, self.quads[:, k]] for k in range(4)]
        e0, e1, e2 = v[1] - v[0], v[2] - v[0], v[3] - v[0]
        n1, n2 = torch.cross(e0, e1, dim=-1), torch.cross(e1, e2, dim=-1)
        l1, l2 = torch.linalg.norm(n1, dim=-1, keepdim=True), torch.linalg.norm(n2, dim=-1, keepdim=True)
        m1, m2 = n1 / l1, n2 / l2
        sign = torch.where(((n1 - n2) * (v[1] - v[3])).sum(-1) > 0, 1.0, -1.0)
        return (e0, e1, e2, l1, l2, m1, m2), (m1 * m2).sum(-1), sign * torch.linalg.norm(torch.cross(m1, m2, dim=-1), dim=-1)

    def update(self):
        a, b, c = (self.X[:, self.tri[:, k]] for k in range(3))
        area = 0.5 * torch.linalg.norm(torch.cross(b - a, c - a, dim=-1), dim=-1)
        self.area = area.sum(1)
        self.volume = (a * torch.cross(b, c, dim=-1)).sum((1, 2)) / 6
        com = ((a + b + c) / 3 * area[..., None]).sum(1) / self.area[:, None]
        shift = torch.zeros_like(com)
        for k, n in enumerate((self.nx, self.ny, self.nz)):
            if self.per[k]:
                shift[:, k] = -n * torch.floor((com[:, k] + 0.5) / n)
        self.com = com + shift
        self.X = self.X + shift[:, None]

    def membrane_forces(self):
        X, prm = self.X, self.prm
        fv = torch.zeros_like(X)

        def add(idx, g):
            fv.index_add_(1, idx, g)

        t0, t1, t2 = (self.tri[:, k] for k in range(3))
        p0, p1, p2 = X[:, t0], X[:, t1], X[:, t2]
        e0, e1 = p1 - p0, p2 - p0
        col = lambda s: s[..., None]  # noqa: E731
        l, lp = torch.linalg.norm(e0, dim=-1), torch.linalg.norm(e1, dim=-1)
        dot = (e0 * e1).sum(-1)
        sp, cp = torch.linalg.norm(torch.cross(e0, e1, dim=-1), dim=-1) / (l * lp), dot / (l * lp)
        l0, l0p, s0, c0 = self.l0, self.l0p, self.sin0, self.cos0
        # the deformation gradient of the triangle, entries a, b, c (c without the stretch of l', as the reference has it)
        A, B, Cc = l / l0, (lp * cp / l0p - l * c0 / l0) / s0, sp / s0
        D11, D22, D12 = (A * A - 1) / 2, (B * B + Cc * Cc - 1) / 2, A * B / 2
        I1 = 2 * (D11 + D22)
        I2 = I1 + 4 * (D11 * D22 - D12 * D12)
        w1, w2 = I1 + 1, prm[1] * I2 - 1
        gl = (-e0 / col(l), e0 / col(l), torch.zeros_like(e0))
        glp = (-e1 / col(lp), torch.zeros_like(e1), e1 / col(lp))
        q1 = e1 / col(l * lp) - col(dot / (l ** 3 * lp)) * e0
        q2 = e0 / col(l * lp) - col(dot / (l * lp ** 3)) * e1
        gc = (-q1 - q2, q1, q2)
        for k, idx in enumerate((t0, t1, t2)):
            g11 = col(l / l0 ** 2) * gl[k]
            g22 = (col(lp / l0p ** 2 - l * cp * c0 / (l0 * l0p)) * glp[k] + col(l * c0 ** 2 / l0 ** 2 - lp * cp * c0 / (l0p * l0)) * gl[k]
                   - col(l * lp * c0 / (l0 * l0p)) * gc[k]) / col(s0 ** 2)
            g12 = (col(lp * cp / l0p - 2 * l * c0 / l0) * gl[k] + col(l * cp / l0p) * glp[k] + col(l * lp / l0p) * gc[k]) / col(2 * l0p * s0)
            gI1 = 2 * (g11 + g22)
            gI2 = col(2 + 4 * D22) * g11 + col(2 + 4 * D11) * g22 - col(8 * D12) * g12
            add(idx, col(-prm[0] / 2 * self.a0) * (col(w1) * gI1 + col(w2) * gI2))
        if self.model != "skalak_bending":
            return fv
        # global area and volume penalties (k_area_global, k_volume), then bending
        n = torch.cross(e0, e1, dim=-1)
        m = n / torch.linalg.norm(n, dim=-1, keepdim=True)
        A0 = self.a0.sum()
        ka = (prm[6] * (A0 - self.area) / A0)[:, None, None]
        kv = (prm[8] * (prm[9] - self.volume) / prm[9] / 6)[:, None, None]
        rel = X - self.com[:, None]
        r = (rel[:, t0], rel[:, t1], rel[:, t2])
        for k, idx in enumerate((t0, t1, t2)):
            b, c = r[(k + 1) % 3], r[(k + 2) % 3]
            add(idx, ka * 0.5 * torch.cross(m, c - b, dim=-1) + kv * torch.cross(b, c, dim=-1))
        (e0, e1, e2, l1, l2, m1, m2), cos, sin = self.angles(X)
        en = torch.linalg.norm(e1, dim=-1, keepdim=True)
        eu = e1 / en
        pre = col(prm[10] * (-self.c0 * sin + self.s0 * cos))
        d = lambda a, b: (a * b).sum(-1, keepdim=True)  # noqa: E731
        q = self.quads
        add(q[:, 0], pre * (d(eu, e1 - e2) / l2 * m2 + d(eu, e1 - e0) / l1 * m1))
        add(q[:, 1], pre * (-en / l1 * m1))
        add(q[:, 2], pre * (d(eu, e2) / l2 * m2 + d(eu, e0) / l1 * m1))
        add(q[:, 3], pre * (-en / l2 * m2))
        return fv

    def interactions(self, fv):
        rng, beta, strength = PIPE_PP
        box = torch.tensor([self.nx, self.ny, self.nz], dtype=F64, device=self.dev)
        flat = self.X.reshape(-1, 3)
        for k in range(self.X.shape[0]):
            near = torch.ones(flat.shape[0], dtype=torch.bool, device=self.dev)
            nv = self.X.shape[1]
            near[k * nv:(k + 1) * nv] = False
            lo, hi = self.X[k].amin(0), self.X[k].amax(0)
            off = flat - 0.5 * (lo + hi)
            off = off - torch.floor(off / box + 0.5) * box
            near &= (off.abs() <= 0.5 * (hi - lo) + rng).all(1)
            other = flat[near]
            if other.shape[0] == 0:
                continue
            dr = other[None] - self.X[k][:, None]
            dr = dr - torch.floor(dr / box + 0.5) * box
            dist = torch.linalg.norm(dr, dim=-1)
            x = torch.exp(beta * (rng - dist))
            phi = torch.where(dist <= rng, 2 * beta * strength * x * (x - 1), torch.zeros_like(x))
            fv[k] += (-(phi / dist)[..., None] * dr).sum(1)
        y, z = self.X[..., 1] - self.pipe[0], self.X[..., 2] - self.pipe[1]
        rr = torch.sqrt(y * y + z * z)
        dist = self.pipe[2] - rr
        phi = torch.where(dist <= PIPE_WALL[0], (PIPE_WALL[0] - dist) * PIPE_WALL[1], torch.zeros_like(rr))
        fv[..., 1] -= phi * y / rr
        fv[..., 2] -= phi * z / rr
        return fv

    def stencil(self):
        """Node indices and weights of every vertex: (vertices, nodes)."""
        p = self.X.reshape(-1, 3)
        s = 4 if self.dirac == "peskin" else 3
        g, w = [], []
        for k, n in enumerate((self.nx, self.ny, self.nz)):
            node = torch.ceil(p[:, k] - s / 2)[:, None] + torch.arange(s, dtype=F64, device=self.dev)
            d = (node - p[:, k:k + 1]).abs()
            if s == 4:
                wt = torch.where(d <= 1, 3 - 2 * d + torch.sqrt((1 + 4 * d * (1 - d)).clamp(min=0)), 5 - 2 * d - torch.sqrt((-7 + 4 * d * (3 - d)).clamp(min=0))) / 8
            else:
                wt = torch.where(d > 0.5, 5 - 3 * d - torch.sqrt((1 - 3 * (1 - d) ** 2).clamp(min=0)), 2 * (1 + torch.sqrt((1 - 3 * d * d).clamp(min=0)))) / 6
            node = node.long()
            if self.per[k]:
                node = node % n
            else:
                wt = torch.where((node >= 0) & (node < n), wt, torch.zeros_like(wt))
                node = node.clamp(0, n - 1)
            g.append(node)
            w.append(wt)
        idx = g[0][:, None, None, :] + self.nx * (g[1][:, None, :, None] + self.ny * g[2][:, :, None, None])
        wt = w[0][:, None, None, :] * w[1][:, None, :, None] * w[2][:, :, None, None]
        return idx.reshape(p.shape[0], -1), wt.reshape(p.shape[0], -1)

    def voxelize(self):
        """Parity of the crossings below each node, along z, of the (one) closed membrane."""
        self.phase = torch.zeros(self.shape, dtype=torch.bool, device=self.dev)
        z = torch.arange(self.nz, dtype=F64, device=self.dev)
        for X in self.X:
            i = torch.arange(math.ceil(X[:, 0].min()), math.floor(X[:, 0].max()) + 1, device=self.dev)
            j = torch.arange(math.ceil(X[:, 1].min()), math.floor(X[:, 1].max()) + 1, device=self.dev)
            px, py = (t.reshape(-1, 1).to(F64) for t in torch.meshgrid(i, j, indexing="ij"))
            a, b, c = (X[self.tri[:, k]] for k in range(3))
            d = (b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (c[:, 0] - a[:, 0]) * (b[:, 1] - a[:, 1])
            u = ((px - a[:, 0]) * (c[:, 1] - a[:, 1]) - (c[:, 0] - a[:, 0]) * (py - a[:, 1])) / d
            v = ((b[:, 0] - a[:, 0]) * (py - a[:, 1]) - (px - a[:, 0]) * (b[:, 1] - a[:, 1])) / d
            hit, tri = torch.nonzero((u >= 0) & (v >= 0) & (u + v <= 1), as_tuple=True)
            h = a[tri, 2] + u[hit, tri] * (b[tri, 2] - a[tri, 2]) + v[hit, tri] * (c[tri, 2] - a[tri, 2])
            count = torch.zeros((px.shape[0], self.nz), dtype=torch.int32, device=self.dev)
            lo = h.min() - 0.5 if h.numel() else 0.0
            zz = torch.remainder(z - lo, self.nz) + lo  # the image of each node above the lowest crossing
            count.index_add_(0, hit, (h[:, None] < zz[None]).to(torch.int32))
            X_, Y_ = (px[:, 0].long() % self.nx), py[:, 0].long()
            self.phase[:, Y_, X_] |= (count % 2 == 1).T

    def step(self):
        u = self.velocity().reshape(3, -1)
        fv = self.membrane_forces()
        if self.pipe is not None:
            fv = self.interactions(fv)
        idx, wt = self.stencil()
        F = torch.zeros_like(u)
        F[0] += self.body
        for a in range(3):
            F[a].index_add_(0, idx.reshape(-1), (wt * fv[..., a].reshape(-1, 1)).reshape(-1))
        vel = torch.stack([(u[a][idx] * wt).sum(1) for a in range(3)], -1)
        self.F = list(F.reshape((3,) + self.shape))
        self.X = self.X + vel.reshape(self.X.shape)
        self.update()
        if self.omega_in is not None:
            self.voxelize()
        self.collide_and_stream()

    def stats(self):
        return torch.cat([self.area[:, None], self.volume[:, None], self.com], 1)


def _exact_coupled(case, w):
    kw = w["lattice"]
    E = _Exact((case["nz"], case["ny"], case["nx"]), kw["omega"], walls=case["walls"], wall_u=U_WALL, body=0.0 if case["walls"] == "shear" else BODY,
               omega_in=kw.get("omega_inner"), pipe=_pipe(case) if case["walls"] == "pipe" else None)
    u = torch.as_tensor(w["u"], device=E.dev)
    E.start(torch.ones(E.shape, dtype=F64, device=E.dev), u)
    E.particles(w, case["dirac"])
    seen = []
    for _ in range(case["steps"]):
        E.step()
        seen.append(E.stats())
    got = [E.velocity(), E.X.reshape(-1, 3), seen[-1]]
    return got + ([torch.stack(seen)] if case["read"] == "step" else [])


def exact(case, seed):
    if case["kind"] == "coupled":
        return _exact_coupled(case, _setup(case, seed))
    if case["kind"] == "batch":
        got = [_exact_coupled(c, w) for c, w in _instances(case, seed)]
        return [torch.cat([g[k].reshape(-1) for g in got]) for k in range(3)]
    tau, coll = (0.8, case["collision"]) if case["kind"] == "lattice" else (TAU, "bgk")
    E = _Exact((case["nz"], case["ny"], case["nx"]), 1 / tau, collision=coll)
    E.start(*_flow(case, seed, E.dev))
    for _ in range(case["steps"]):
        E.collide_and_stream()
    return [E.velocity() if case["kind"] == "lattice" else E.f.permute(3, 2, 1, 0).contiguous()]
