"""Membranes with link springs in FP32 (element kernels, one particle's elements over several CTAs) against FP64:
one CTA and several per particle, one particle and several, different block sizes.  1e-3 of the largest force:
FP32 positions relative to the centre give edges to 1e-6, under strains of 5 per cent."""
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


@pytest.mark.parametrize("block", [0, 64, 512])
@pytest.mark.parametrize("level,cells", [(1, 1), (3, 1), (3, 3), (4, 2)])
def test_link_spring_forces_fp32(ctx, level, cells, block):
    rng = np.random.default_rng(4)
    xyz, tri = meshes.icosphere(level, 6.0)
    L0 = np.linalg.norm(xyz[tri[:, 0]] - xyz[tri[:, 1]], axis=1).mean()
    prm = bib.membrane_params(shear_modulus=1e-2, L0=L0, k_area_global=0.1, k_area_local=0.1, k_volume=0.1, k_bend=1e-3, vol_desired=880.0)
    pos = [xyz * np.array([1.05, 0.97, 1.02]) + 0.01 * L0 * rng.standard_normal(xyz.shape) + np.array([10.0 + 14 * k, 15.0, 16.0])
           for k in range(cells)]
    out = []
    for storage in ("f64", "f32"):
        lat = ctx.add_domain(48, 32, 32, omega=1.0, storage=storage)
        lat.set_tuning(membrane_block=block)
        shapes = bib.ParticleShapeLibrary(ctx)
        fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes)
        sid = shapes.store_mesh(xyz, tri, "m")
        for p in pos:
            fsi.add_particle(sid, "rbc_wlcpow", prm, p)
        fsi.ibm_step()
        out.append(np.concatenate([fsi.get_particle(k)["force"] for k in range(cells)]))
    assert np.abs(out[0]).max() > 1e-4
    assert np.abs(out[1] - out[0]).max() <= 1e-3 * np.abs(out[0]).max()
