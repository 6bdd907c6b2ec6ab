"""Spreading by rows against the oracle's spreading: both kernels, FP64 and FP32 fields, every alignment
of a row (nx = 1, 2, 3 mod 4), supports that wrap along x, walled axes, and
vertex counts around a multiple of 32.  FP64 to 1e-13 and FP32 to 5e-6 of the largest spread force (three
weights off by 1e-7 of the largest each, two products and the sum of up to about 20 vertices per cell)."""
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


@pytest.mark.parametrize("storage,tol", [("f64", 1e-13), ("f32", 5e-6)])
@pytest.mark.parametrize("dirac", ["roma", "peskin"])
@pytest.mark.parametrize("dims,periodic,level,offset", [((13, 12, 11), (1, 1, 1), 1, -1.0), ((14, 16, 12), (1, 0, 1), 2, -1.0),
                                                        ((15, 13, 16), (1, 0, 0), 0, -1.0), ((5, 12, 12), (1, 1, 1), 1, -1.0)])
def test_spread_rows_match_oracle(ctx, dims, periodic, level, offset, dirac, storage, tol):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    walls = {"wall_y": "none" if periodic[1] else "halfway_bb", "wall_z": "none" if periodic[2] else "halfway_bb"}
    xyz, tri = meshes.icosphere(level, 3.3)
    pos = meshes.place(1.05 * xyz, None, (0.2, ny / 2 - 1.7, nz / 2 + 1.9))
    prm = bib.membrane_params(G=1e-2, C=1.0)
    lat = ctx.add_domain(nx, ny, nz, periodic=periodic, omega=1.0, storage=storage, **walls)
    shapes = bib.ParticleShapeLibrary(ctx)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac, field_offset=offset)
    pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", prm, pos)
    fsi.ibm_step()
    force = fsi.get_particle(pid)["force"]  # the library's own: the spreading alone is compared
    L = O.lattice(dims, periodic, "bgk_guo_vof", 1.0, 1.0, **walls)
    want, got = O.spread(L, dirac, pos, force, offset=offset), lat.get_external_force()
    assert np.abs(want).max() > 1e-5
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("dirac", ["roma", "peskin"])
def test_positive_field_offset_leaves_the_same_nodes_out(ctx, dirac):
    """With a positive field offset the periodic remap leaves nodes at the upper faces out; the
    deterministic spreading, node by node, says which (FP64, 1e-13 of the largest force)."""
    xyz, tri = meshes.icosphere(1, 3.3)
    pos = meshes.place(1.05 * xyz, None, (0.2, 4.3, 7.9))
    F = []
    for spread in ("atomic", "deterministic"):
        lat = ctx.add_domain(16, 12, 12, omega=1.0)
        shapes = bib.ParticleShapeLibrary(ctx)
        fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac, field_offset=2.0, spread=spread)
        fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", bib.membrane_params(G=1e-2, C=1.0), pos)
        fsi.ibm_step()
        F.append(lat.get_external_force())
    assert np.abs(F[1]).max() > 1e-5
    assert np.abs(F[0] - F[1]).max() <= 1e-13 * np.abs(F[1]).max()
