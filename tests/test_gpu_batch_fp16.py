"""FP16 batches (packed pairs of cells, the reset of the previous force with one body force after another) against
single lattices: nine steps, populations to 5e-5 (a unit in the last place of f-bar up to 0.004 is 1.9e-6 a step, and
what follows from it), positions to 2e-4 (velocity fields in 2^-11 of 0.02, nine steps, and the populations')."""
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


def lattices(ctx, dirac, lam):
    out = []
    for k, (dims, body, fd) in enumerate([((32, 30, 28), 0.0, True), ((48, 24, 25), 2e-6, False), ((40, 40, 24), -1e-6, False),
                                          ((8, 26, 26), 2e-6, False), ((512, 12, 13), 0.0, True)]):
        nx, ny, nz = dims
        kw = dict(use_phase=True, omega_inner=1 / 1.3) if lam else {}
        kw.update(dict(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=[[-0.02, 0, 0], [0.02, 0, 0], [0, 0, 0], [0, 0, 0]]) if fd
                  else dict(periodic=(1, 1, 1), body_force=(body, -body, 2 * body)))
        lat = ctx.add_domain(nx, ny, nz, omega=1.1, storage="f16", **kw)
        u0 = np.zeros((3, nz, ny, nx))
        u0[0] = (0.02 * (2 * np.arange(ny) / (ny - 1) - 1))[None, :, None] if fd else 0.01
        lat.initialize_at_equilibrium(None, u0)
        xyz, tri = meshes.icosphere(2, min(3.4, min(dims) / 4))
        shapes = bib.ParticleShapeLibrary(ctx)
        fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, dirac=dirac)
        pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", bib.membrane_params(G=1e-3, C=1.0),
                               meshes.place(1.05 * xyz, None, (0.4 + k, ny / 2 + 0.2, nz / 2 - 0.3)))
        out.append((lat, fsi, pid))
    return out


@pytest.mark.parametrize("dirac", ["roma", "peskin"])
@pytest.mark.parametrize("lam", [False, True])
def test_fp16_batch_equals_individual_steps(ctx, dirac, lam):
    solo, grouped = lattices(ctx, dirac, lam), lattices(ctx, dirac, lam)
    batch = bib.Batch(ctx, [g[0] for g in grouped])
    batch.step(5)  # odd: graph pairs plus one plain step
    batch.step(4)
    for (ls, fs, ps), (lg, fg, pg) in zip(solo, grouped):
        fs.step(9)
        a, b = fs.get_particle(ps), fg.get_particle(pg)
        assert np.isfinite(b["pos"]).all()
        assert np.abs(a["pos"] - b["pos"]).max() <= 2e-4
        assert np.abs(ls.receive() - lg.receive()).max() <= 5e-5
        lg.check_health()
    batch.close()
