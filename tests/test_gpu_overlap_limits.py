"""Coupled steps on both sides of the limits up to which membranes run beside the collision (support nodes against
cells, per storage, model and collision kernel), against the consecutive steps that profiling forces, from the same
state.  The two form the velocity by different kernels in the storage's compute type and agree to its rounding: after
six steps positions to 1e-12 (FP64), 1e-7 (FP32: velocities of 0.02 to 1e-7 of their value and the forces that follow),
1e-4 (FP16 velocity field: 0.02 to 2^-11 each step)."""
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


# cells of 642 (level 3) or 162 vertices (level 2): nodes below and above the limit of 64 x 48 x 48 cells
CASES = [("f16", 64, "skalak_bending", 3, (2, 3)), ("f32", 64, "skalak_bending", 3, (2, 3)), ("f32", 64, "rbc_wlcpow", 3, (2, 3)),
         ("f64", 64, "capsule_skalak", 3, (1, 2)), ("f64", 64, "skalak_bending", 2, (1, 2)), ("f64", 63, "skalak_bending", 3, (1, 4)),
         ("f64", 64, "skalak_bending", 4, (1,))]


@pytest.mark.parametrize("storage,nx,model,level,counts", CASES)
def test_both_sides_of_the_limit(ctx, storage, nx, model, level, counts):
    ny, nz = 48, 48
    u0 = np.zeros((3, nz, ny, nx))
    u0[0] = (0.02 * (2 * np.arange(ny) / (ny - 1) - 1))[None, :, None]
    xyz, tri = meshes.icosphere(level, 5.0)
    prm = dict(G=2e-3, C=1.0) if model != "rbc_wlcpow" else dict(shear_modulus=2e-3, L0=0.8)
    prm = bib.membrane_params(**prm, k_area_global=0.1, k_volume=0.1, vol_desired=520.0, k_bend=1e-4)
    for cells in counts:
        ends = []
        for profiled in (False, True):
            lat = ctx.add_domain(nx, ny, nz, omega=0.9, storage=storage, periodic=(1, 0, 1), wall_y="fd_velocity",
                                 wall_u=[[-0.02, 0, 0], [0.02, 0, 0], [0, 0, 0], [0, 0, 0]])
            lat.initialize_at_equilibrium(None, u0)
            shapes = bib.ParticleShapeLibrary(ctx)
            fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, spread="deterministic")
            sid = shapes.store_mesh(xyz, tri, "c")
            for k in range(cells):
                fsi.add_particle(sid, model, prm, xyz * np.array([1.05, 0.96, 1.0]) + np.array([7.3 + 13 * k, 24.2, 23.7]))
            ctx.set_profiling(profiled)
            try:
                fsi.step(6)
            finally:
                ctx.set_profiling(False)
            ends.append(np.concatenate([fsi.get_particle(k)["pos"] for k in range(cells)]))
        assert np.abs(ends[0] - ends[1]).max() <= {"f64": 1e-12, "f32": 1e-7, "f16": 1e-4}[storage]
