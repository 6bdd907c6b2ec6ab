"""The velocity field at the vertices' support nodes only (one capsule in a large lattice with a phase
field, or the immersed-boundary step alone) against the oracle: periodic images, walls and both
kernels.  FP64 vertex velocities to 1e-13 of the largest (the interpolation's summation order and fused
multiply-adds over 64 products)."""
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


@pytest.mark.parametrize("dirac", ["roma", "peskin"])
@pytest.mark.parametrize("dims,walls,at", [((41, 40, 40), "none", (0.3, 39.6, 0.2)), ((48, 37, 40), "shear", (20.2, 4.1, 39.7)),
                                           ((40, 41, 41), "channel", (39.9, 36.4, 4.2))])
def test_support_velocity_matches_oracle(ctx, dirac, dims, walls, at):
    nx, ny, nz = dims
    kw = {"none": dict(periodic=(1, 1, 1)),
          "shear": dict(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=[[-0.02, 0, 0], [0.02, 0, 0], [0, 0, 0], [0, 0, 0]]),
          "channel": dict(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb")}[walls]
    rng = np.random.default_rng(3)
    u0 = rng.uniform(-0.02, 0.02, (3, nz, ny, nx))
    xyz, tri = meshes.icosphere(2, 4.0)
    pos = meshes.place(xyz, meshes.random_rotation(rng), at)
    prm = bib.membrane_params(G=1e-3, C=1.0)
    lat = ctx.add_domain(nx, ny, nz, omega=1.0, **kw)
    lat.initialize_at_equilibrium(None, u0)
    f0 = lat.receive()
    shapes = bib.ParticleShapeLibrary(ctx)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac)
    pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", prm, pos)
    fsi.ibm_step()  # velocity at the support nodes, interpolation, move
    L = O.lattice(dims, kw["periodic"], "bgk_guo_vof", 1.0, 1.0, wall_y=kw.get("wall_y", "none"), wall_z=kw.get("wall_z", "none"),
                  wall_u=kw.get("wall_u"))
    S = O.System(L, dirac, -1.0)
    S.f[...] = f0
    opid = S.add_particle(S.add_shape(xyz, tri), "capsule_skalak", prm, pos)
    S.step(1)  # the coupled step interpolates the same velocity
    want, got = S.particle(opid)["vel"], fsi.get_particle(pid)["vel"]
    assert np.abs(want).max() > 1e-3
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
