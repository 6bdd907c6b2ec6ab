"""Spreading with a pipe boundary: a vertex away from the wall is spread by rows like any other, near the
wall the 2-point TopHat takes the share 1 - w of its force.  Against the oracle's spreading of w times the
force plus the TopHat restated here (FP64 1e-13, FP32 5e-6 of the largest: weights off by 1e-7 of the largest
each, two products and a sum of up to 20 vertices per cell), and bit for bit against a lattice without a
boundary where no vertex is near the wall (one vertex per support: nothing depends on the order)."""
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


def spread(ctx, storage, dirac, dims, xyz, tri, pos, pipe, batch=False):
    lat = ctx.add_domain(*dims, omega=1.0, storage=storage)
    shapes = bib.ParticleShapeLibrary(ctx)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac)
    pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", bib.membrane_params(G=1e-2, C=1.0), pos)
    if pipe is not None:
        fsi.set_boundary(*pipe)
    fsi.ibm_step()
    return fsi.get_particle(pid)["force"], lat.get_external_force()


def tophat(dims, pos, force):
    nx, ny, nz = dims
    F = np.zeros((3, nz, ny, nx))
    lo = np.ceil(pos - 1.0).astype(int)
    for v in range(len(pos)):
        for m in np.ndindex(2, 2, 2):
            node = lo[v] + m
            w = np.prod(1.0 - np.abs(node - pos[v]))
            F[:, node[2] % nz, node[1] % ny, node[0] % nx] += w * force[v]
    return F


@pytest.mark.parametrize("storage,tol", [("f64", 1e-13), ("f32", 5e-6), ("f16", 5e-6)])
@pytest.mark.parametrize("dirac,h", [("roma", 1.5), ("peskin", 2.0)])
@pytest.mark.parametrize("dims,level,shift", [((14, 22, 22), 2, 1.7), ((13, 21, 23), 1, 3.0), ((30, 22, 22), 3, 0.4)])
def test_near_wall_blend_matches_oracle(ctx, dims, level, shift, dirac, h, storage, tol):
    nx, ny, nz = dims
    xyz, tri = meshes.icosphere(level, 5.0)
    y0, z0, R = 0.5 * (ny - 1), 0.5 * (nz - 1), 8.9
    pos = meshes.place(1.05 * xyz, None, (0.3, y0 + shift, z0 - 0.2))
    force, got = spread(ctx, storage, dirac, dims, xyz, tri, pos, (y0, z0, R))
    w = np.clip(R - np.hypot(pos[:, 1] - y0, pos[:, 2] - z0) - h, 0.0, 1.0)[:, None]
    assert (w == 1).any() and (w < 1).any() == (shift > 1)  # the last one reaches no blend
    L = O.lattice(dims, (1, 1, 1), "bgk_guo_vof", 1.0, 1.0)
    want = O.spread(L, dirac, pos, w * force, offset=-1.0) + tophat(dims, pos, (1 - w) * force)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("dirac", ["roma", "peskin"])
def test_vertices_away_from_the_wall_are_spread_as_without_one(ctx, dirac, storage):
    xyz, tri = meshes.icosphere(0, 6.5)  # 12 vertices, 6.8 apart: no two share a node
    pos = meshes.place(1.03 * xyz, None, (11.7, 12.2, 11.4))
    out = [spread(ctx, storage, dirac, (24, 24, 24), xyz, tri, pos, pipe) for pipe in (None, (12.0, 12.0, 40.0))]
    assert np.abs(out[0][1]).max() > 1e-5
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
