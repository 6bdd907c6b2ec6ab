"""Coupled steps whose membranes run beside the collision (few vertices in the lattice) against the oracle
over graph pairs, single steps and eager steps mixed, with forces read in between; FP64 populations to 1e-14
and positions to 1e-11 (the sums' order and fused multiply-adds over a few steps).  The three ways of issuing
steps give the same bits with deterministic spreading."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")
from biblbm_gb300 import meshes  # noqa: E402


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


def system(ctx, dims, walls, level, dirac, storage, spread, at=None):
    nx, ny, nz = dims
    U = [[-0.02, 0, 0], [0.02, 0, 0], [0, 0, 0], [0, 0, 0]]
    kw = dict(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=U) if walls == "fd" else dict(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb")
    xyz, tri = meshes.icosphere(level, 4.0)
    pos = meshes.place(xyz * np.array([1.1, 0.95, 1.0]), None, (0.4, ny / 2 if at is None else at, nz / 2 + 0.3))
    prm = bib.membrane_params(G=5e-3, C=1.0, k_area_global=0.1, k_volume=0.1, vol_desired=260.0, k_bend=1e-3)
    u0 = np.zeros((3, nz, ny, nx))
    u0[0] = (0.02 * (2 * np.arange(ny) / (ny - 1) - 1))[None, :, None]
    lat = ctx.add_domain(nx, ny, nz, omega=0.9, storage=storage, **kw)
    lat.initialize_at_equilibrium(None, u0)
    shapes = bib.ParticleShapeLibrary(ctx)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac, spread=spread)
    pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "skalak_bending", prm, pos)
    return lat, fsi, pid, kw, xyz, tri, prm, pos


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("dims,walls,level,dirac", [((33, 25, 24), "fd", 1, "roma"), ((24, 24, 26), "channel", 1, "peskin"),
                                                    ((40, 24, 24), "fd", 2, "roma")])
def test_ways_of_stepping_agree(ctx, storage, dims, walls, level, dirac):
    ends = []
    for way in ("pairs", "single", "mixed", "eager"):
        lat, fsi, pid, *_ = system(ctx, dims, walls, level, dirac, storage, "deterministic")
        ctx.set_graph_mode(way != "eager")
        try:
            if way == "single":
                for _ in range(7):
                    fsi.step(1)
            elif way == "mixed":
                for k in (3, 1, 2, 1):
                    fsi.step(k)
                    fsi.get_particle(pid)
            else:
                fsi.step(7)
        finally:
            ctx.set_graph_mode(True)
        p = fsi.get_particle(pid)
        ends.append((lat.receive(), p["pos"], p["force"], p["vel"], lat.get_external_force()))
    for e in ends[1:]:
        for a, b in zip(ends[0], e):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("dims,walls,level,dirac,at", [((33, 25, 24), "fd", 1, "roma", None), ((24, 24, 26), "channel", 1, "peskin", None),
                                                       ((33, 25, 24), "fd", 1, "roma", 5.0), ((33, 25, 24), "fd", 1, "peskin", 18.6)])
def test_overlapped_steps_match_oracle(ctx, dims, walls, level, dirac, at):
    lat, fsi, pid, kw, xyz, tri, prm, pos = system(ctx, dims, walls, level, dirac, "f64", "atomic", at)
    f0 = lat.receive()
    L = O.lattice(dims, kw["periodic"], "bgk_guo_vof", 0.9, 0.9, wall_y=kw.get("wall_y", "none"), wall_z=kw.get("wall_z", "none"),
                  wall_u=kw.get("wall_u"))
    S = O.System(L, dirac, -1.0)
    S.f[...] = f0
    opid = S.add_particle(S.add_shape(xyz, tri), "skalak_bending", prm, pos)
    for k in (2, 1, 4):
        S.step(k)
        fsi.step(k)
        g, w = fsi.get_particle(pid), S.particle(opid)
        assert np.abs(lat.receive() - S.f).max() < 1e-14
        assert np.abs(g["pos"] - w["pos"]).max() < 1e-11
        assert np.abs(g["force"] - w["force"]).max() < 1e-8 * np.abs(w["force"]).max()


@pytest.mark.parametrize("kernel", ["auto", "rows"])
@pytest.mark.parametrize("dims,level", [((32, 24, 24), 1), ((27, 24, 26), 1)])
def test_cell_types_beside_the_fluid(ctx, kernel, dims, level):
    """Support nodes in bounce-back and no-dynamics cells: the profiled (consecutive) steps' values."""
    nx, ny, nz = dims
    types = np.zeros((nz, ny, nx), np.uint8)
    types[:, :3] = 2
    types[:, -3:] = 2
    types[2, 3:6] = 1
    ends = []
    for profiled in (False, True):
        lat = ctx.add_domain(nx, ny, nz, omega=1.1, body_force=(1e-5, 0, 0))
        lat.set_cell_types(types)
        lat.set_tuning(kernel=kernel)
        lat.initialize_at_equilibrium(None, 0.01 * np.ones((3, nz, ny, nx)))
        xyz, tri = meshes.icosphere(level, 4.0)
        pos = meshes.place(xyz, None, (3.0, 6.7, 5.0))
        shapes = bib.ParticleShapeLibrary(ctx)
        fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, spread="deterministic")
        pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", bib.membrane_params(G=5e-3, C=1.0), pos)
        ctx.set_profiling(profiled)
        try:
            fsi.step(5)
        finally:
            ctx.set_profiling(False)
        p = fsi.get_particle(pid)
        ends.append((lat.receive(), p["pos"], p["vel"]))
    for a, b, tol in zip(ends[0], ends[1], (1e-14, 1e-12, 1e-13)):
        assert np.abs(a - b).max() <= tol
