"""Wall interactions of FP32 and FP16 lattices keep their FP64 bits in the vertex forces: for a membrane at
rest, whose own forces vanish to FP32 rounding (6e-8 of the modulus, far below 1e-15 of the wall force for
the modulus here), the vertex forces are those of an FP64 lattice to 1e-14 of the largest (the FP64
evaluation alone: a sum of three decorators)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")
from biblbm_gb300 import meshes  # noqa: E402


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


def forces(ctx, storage, spread, cells):
    lat = ctx.add_domain(32, 24, 24, omega=1.0, storage=storage)
    shapes = bib.ParticleShapeLibrary(ctx)
    xyz, tri = meshes.icosphere(2, 4.0)
    sid = shapes.store_mesh(xyz, tri, "m")
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, spread=spread)
    for k in range(cells):
        fsi.add_particle(sid, "capsule_skalak", bib.membrane_params(G=1e-14, C=1.0), xyz + np.array([5.3 + 0.1 * k, 6.1, 12.2]))
    fsi.add_wall_interaction(bib.SpringPotential(9.0, 1e-2), 1, 0.0, 23.0)
    fsi.add_wall_interaction(bib.MorsePotential(12.0, 0.3, 1e-2), 2, 0.0, 23.0)
    fsi.add_pipe_wall_interaction(bib.SpringPotential(20.0, 1e-3), 11.5, 11.5, 12.0)
    fsi.ibm_step()
    return np.concatenate([fsi.get_particle(k)["force"] for k in range(cells)])


@pytest.mark.parametrize("spread", ["atomic", "deterministic"])
@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("cells", [1, 3])
def test_wall_forces_keep_their_bits(ctx, storage, spread, cells):
    want = forces(ctx, "f64", "deterministic", cells)
    got = forces(ctx, storage, spread, cells)
    assert np.abs(want).min() > 1e-6 * np.abs(want).max() or np.abs(want).max() > 1e-3
    assert np.abs(got - want).max() <= 1e-14 * np.abs(want).max()
