"""Collide-and-stream over linear tiles (rows no row tile takes) against the direct kernels on the same
state: odd rows, even rows that are no multiple of 16 bytes, rows longer than a tile, the last partial
tile; periodic, halfway and finite-difference walls, moving walls, cell types, a phase field, all
collisions, lattice-only and coupled.  One step: FP32 to 2e-8 (populations below 0.02, a few roundings of
6e-8 each), FP16 to one unit in the last place of the largest (0.02 * 8192 = 164: 0.125 / 8192)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")

U = [[0.01, 0, 0.005], [-0.02, 0, 0], [0.01, 0.003, 0], [0, 0, 0]]
SETUP = {
    "periodic_trt": dict(kw=dict(periodic=(1, 1, 1), collision="trt")),
    "periodic_bgk": dict(kw=dict(periodic=(1, 1, 1), collision="bgk")),
    "channel": dict(kw=dict(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb", wall_u=U, body_force=(1e-5, 0, -2e-5))),
    "fd": dict(kw=dict(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=U, body_force=(1e-5, 0, 0))),
    "phase_types": dict(kw=dict(periodic=(1, 1, 0), wall_z="halfway_bb", use_phase=True, omega_inner=0.7), types=True),
}
DIMS = {"f32": [(83, 81, 79), (523, 33, 31), (514, 32, 33)], "f16": [(35, 33, 31), (34, 32, 31), (520, 9, 8), (1024, 6, 7)]}


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("setup", list(SETUP))
@pytest.mark.parametrize("storage,dims", [(s, d) for s in DIMS for d in DIMS[s]])
def test_linear_tiles_match_direct_kernels(ctx, storage, dims, setup, coupled):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + ny)
    f0, F0 = rng.uniform(-0.018, 0.018, (19, nz, ny, nx)), rng.uniform(-1e-4, 1e-4, (3, nz, ny, nx))
    out = []
    for kernel in ("auto", "rows"):
        lat = ctx.add_domain(nx, ny, nz, omega=1.2, storage=storage, **SETUP[setup]["kw"])
        lat.set_tuning(kernel=kernel)
        if SETUP[setup].get("types"):
            g = np.random.default_rng(1)
            lat.set_cell_types(g.choice([0, 0, 0, 0, 1, 2], (nz, ny, nx)))
            lat.set_phase(g.integers(0, 2, (nz, ny, nx)).astype(float))
        lat.send(f0)
        lat.set_external_force(F0)
        if coupled:
            fsi = bib.ImmersedBoundaryDynamics3D(lat, bib.ParticleShapeLibrary(ctx))
            fsi.step(1)
            F = lat.get_external_force()
        else:
            lat.collide_and_stream(1)
            F = F0
        lat.check_health()
        out.append((lat.receive(), F))
    tol = 2e-8 if storage == "f32" else 0.126 / 8192
    assert np.abs(out[0][0]).max() > 0.005
    assert np.abs(out[0][0] - out[1][0]).max() <= tol
    assert np.array_equal(out[0][1], out[1][1])


def test_previous_force_is_reset(ctx):
    """Two coupled steps with a body force and no particles: the force field is the body force."""
    lat = ctx.add_domain(35, 33, 31, periodic=(1, 1, 1), storage="f16", body_force=(1e-5, -2e-5, 3e-5))
    fsi = bib.ImmersedBoundaryDynamics3D(lat, bib.ParticleShapeLibrary(ctx))
    lat.set_external_force(np.ones((3, 31, 33, 35)))
    fsi.step(3)
    body = np.array([1e-5, -2e-5, 3e-5], dtype=np.float32).astype(float)[:, None, None, None]
    assert np.array_equal(lat.get_external_force(), np.broadcast_to(body, (3, 31, 33, 35)))
