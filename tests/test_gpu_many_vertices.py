"""Interpolation by one thread per vertex, which lattices and batches of more than 24,576 vertices take, in its
variants: both delta kernels, all storage types, batches, the sparse reset's share of the previous force and a pipe
boundary; spheres of 2562 vertices, nine below the line and ten above it.

FP64 to 1e-13 of the largest velocity (27 or 64 products in another order), FP32 to 2e-6 (weights to 1e-7 of the
largest each, and the sum), FP16 to 1e-3 (its velocity field, 2^-11)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")
from biblbm_gb300 import meshes  # noqa: E402

TOL = {"f64": 1e-13, "f32": 2e-6, "f16": 1e-3}


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


def lattice(ctx, dims, storage, cells, dirac="roma", G=0.0, first=0, spread="atomic", radius=6.0, **kw):
    nx, ny, nz = dims
    lat = ctx.add_domain(nx, ny, nz, omega=1.1, storage=storage, **kw)
    rng = np.random.default_rng(8)
    X, Y, Z = (2 * np.pi * np.arange(n) / n for n in dims)
    u = 0.02 * np.stack([np.sin(X)[None, None, :] * np.cos(Y)[None, :, None] * np.cos(Z)[:, None, None] for _ in range(3)])
    u *= np.array([1.0, -0.7, 0.4])[:, None, None, None]
    lat.initialize_at_equilibrium(None, u)
    shapes = bib.ParticleShapeLibrary(ctx)
    xyz, tri = meshes.icosphere(4, radius)
    sid = shapes.store_mesh(xyz, tri, "c")
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac, spread=spread)
    at = rng.uniform(0.0, 1.0, (24, 3)) * np.array([nx, ny - 15.0, nz - 15.0]) + np.array([0.0, 7.5, 7.5])
    pos = [meshes.place(1.03 * xyz, None, tuple(at[first + k])) for k in range(cells)]
    for p in pos:
        fsi.add_particle(sid, "capsule_skalak", bib.membrane_params(G=G, C=1.0), p)
    return lat, fsi, pos


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("dirac", ["roma", "peskin"])
@pytest.mark.parametrize("cells", [9, 10])
@pytest.mark.parametrize("walls", ["none", "channel"])
def test_interpolation_matches_oracle(ctx, storage, dirac, cells, walls):
    dims = (40, 29, 27)
    kw = dict(periodic=(1, 1, 1)) if walls == "none" else dict(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb")
    lat, fsi, pos = lattice(ctx, dims, storage, cells, dirac, **kw)
    u = lat.compute_velocity()
    fsi.ibm_step()
    L = O.lattice(dims, kw["periodic"], "bgk_guo_vof", 1.1, 1.1, wall_y=kw.get("wall_y", "none"), wall_z=kw.get("wall_z", "none"))
    for k in range(cells):
        g = fsi.get_particle(k)
        want = O.interpolate(L, dirac, u, pos[k], offset=-1.0)
        assert np.abs(g["vel"] - want).max() <= TOL[storage] * np.abs(u).max()
        assert np.abs(g["pos"] - (pos[k] + g["vel"])).max() <= 1e-14 * 64


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("dirac", ["roma", "peskin"])
def test_batch_above_the_line_matches_lattices_below_it(ctx, storage, dirac):
    dims = (40, 24, 24)
    kw = dict(periodic=(1, 0, 1), wall_y="halfway_bb", body_force=(1e-6, 0, 0))
    solo = [lattice(ctx, dims, storage, 4, dirac, 0.0, 4 * k, **kw) for k in range(3)]
    group = [lattice(ctx, dims, storage, 4, dirac, 0.0, 4 * k, **kw) for k in range(3)]
    batch = bib.Batch(ctx, [g[0] for g in group])
    batch.step(3)
    for _, fsi, _ in solo:
        fsi.step(3)
    for (la, fa, _), (lb, fb, _) in zip(solo, group):
        for k in range(4):
            a, b = fa.get_particle(k), fb.get_particle(k)
            assert np.abs(a["vel"] - b["vel"]).max() <= 3 * TOL[storage] * 0.02
            assert np.abs(a["pos"] - b["pos"]).max() <= 9 * TOL[storage] * 0.02 + 1e-14 * 64
    batch.close()


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("dirac", ["roma", "peskin"])
def test_pipe_boundary_above_the_line(ctx, storage, dirac):
    """Ten spheres, some across the near-wall zone, against two lattices of five."""
    dims, pipe = (40, 30, 30), (14.5, 14.5, 13.7)
    lat, fsi, pos = lattice(ctx, dims, storage, 10, dirac, periodic=(1, 1, 1))
    fsi.set_boundary(*pipe)
    fsi.ibm_step()
    r = np.concatenate([np.hypot(p[:, 1] - pipe[0], p[:, 2] - pipe[1]) for p in pos])
    assert (r > pipe[2] - 1.5).any() and (r < pipe[2] - 3.0).any()
    for half in (0, 1):
        l2, f2, _ = lattice(ctx, dims, storage, 5, dirac, 0.0, 5 * half, periodic=(1, 1, 1))
        f2.set_boundary(*pipe)
        f2.ibm_step()
        for k in range(5):
            a, b = fsi.get_particle(5 * half + k), f2.get_particle(k)
            assert np.abs(a["vel"] - b["vel"]).max() <= TOL[storage] * 0.02
            assert np.abs(a["pos"] - b["pos"]).max() <= 3 * TOL[storage] * 0.02 + 1e-14 * 64


@pytest.mark.parametrize("dirac", ["roma", "peskin"])
def test_sparse_reset_above_the_line(ctx, dirac):
    """Three FP32 steps, sparse against dense; the forces of the strained spheres enter the second step's velocity by
    half of 1e-4 and the bounds are its FP32 rounding over the steps."""
    out = []
    for reset in ("dense", "sparse"):
        lat, fsi, _ = lattice(ctx, (40, 32, 32), "f32", 10, dirac, 1e-4, spread="deterministic", periodic=(1, 1, 1))
        lat.set_tuning(force_reset=reset)
        fsi.step(3)
        out.append((lat.receive(), np.concatenate([fsi.get_particle(k)["pos"] for k in range(10)])))
    assert np.abs(out[0][0] - out[1][0]).max() <= 2e-7
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-6
