"""Membrane forces by patches (FP32 storage) against the FP32 element kernels on the same state, which a
lattice takes when one of its particles has link springs: every patched model, patch counts from one to
many, a last patch of one vertex, open meshes and meshes whose triangles are not all wound alike (their
volume gradient depends on the origin, which both take at the centre), particles of different shapes and a
wall interaction.  1e-4 of the largest force: FP32 positions relative to the centre (6e-8 of the radius)
under strains of a few per cent.  The same bits on every run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")
from biblbm_gb300 import meshes  # noqa: E402

MODELS = {"capsule_neohookean": dict(G=1e-2), "capsule_skalak": dict(G=1e-2, C=1.0),
          "skalak_bending": dict(G=1e-2, C=1.0, k_area_global=1.0, k_area_local=0.1, k_volume=1.0, k_bend=0.05)}


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


def mesh(name):
    if name == "one_patch":
        return meshes.icosphere(0, 5.0)
    if name in ("sphere", "turned", "open"):
        xyz, tri = meshes.icosphere(3, 5.0)
        tri = tri.copy()
        if name == "turned":  # every third triangle wound the other way
            tri[::3] = tri[::3, ::-1]
        if name == "open":  # a cap cut off
            keep = xyz[tri].mean(axis=1)[:, 2] < 3.0
            used = np.unique(tri[keep])
            new = np.full(xyz.shape[0], -1)
            new[used] = np.arange(used.size)
            xyz, tri = xyz[used], new[tri[keep]]
        return xyz, tri
    # 33 vertices: a ring of 31 between two poles, the last patch owns one vertex
    a = 2 * np.pi * np.arange(31) / 31
    ring = np.stack([5 * np.cos(a), 5 * np.sin(a), np.zeros(31)], 1)
    xyz = np.concatenate([ring, [[0, 0, 3.0], [0, 0, -3.0]]])
    nxt = (np.arange(31) + 1) % 31
    tri = np.concatenate([np.stack([np.arange(31), nxt, np.full(31, 31)], 1), np.stack([nxt, np.arange(31), np.full(31, 32)], 1)])
    return xyz, tri


def forces(ctx, storage, parts, spread, wall):
    lat = ctx.add_domain(40, 32, 32, omega=1.0, storage=storage)
    shapes = bib.ParticleShapeLibrary(ctx)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, spread=spread)
    for k, (xyz, tri, model, prm, pos) in enumerate(parts):
        fsi.add_particle(shapes.store_mesh(xyz, tri, "m%d" % k), model, prm, pos)
    if wall:
        fsi.add_wall_interaction(bib.SpringPotential(9.0, 1e-3), 1, 0.0, 31.0)
    fsi.ibm_step()
    return [fsi.get_particle(k)["force"] for k in range(len(parts))]


@pytest.mark.parametrize("name", ["one_patch", "ring33", "sphere", "turned", "open"])
@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("spread", ["atomic", "deterministic"])
def test_patch_forces_match_element_kernels(ctx, name, model, spread):
    rng = np.random.default_rng(2)
    parts = []
    for nm, at in ((name, (12.0, 14.0, 16.0)), ("sphere", (28.0, 17.0, 15.0))):
        xyz, tri = mesh(nm)
        v = float(np.abs(np.einsum("ij,ij->i", xyz[tri[:, 0]], np.cross(xyz[tri[:, 1]], xyz[tri[:, 2]])).sum() / 6))
        prm = bib.membrane_params(**{**MODELS[model], "vol_desired": v})
        pos = xyz * np.array([1.05, 0.97, 1.02]) + 0.02 * rng.standard_normal(xyz.shape) + np.array(at)
        parts.append((xyz, tri, model, prm, pos))
    xyz, tri = meshes.icosphere(1, 2.0)
    springs = (xyz, tri, "rbc_wlcpow", bib.membrane_params(shear_modulus=1e-4, L0=1.0), xyz + np.array([4.0, 4.0, 4.0]))
    want = forces(ctx, "f32", parts + [springs], "deterministic", True)
    got, again = forces(ctx, "f32", parts, spread, True), forces(ctx, "f32", parts, spread, True)
    for w, g, a in zip(want, got, again):
        assert np.abs(w).max() > 1e-5
        assert np.abs(g - w).max() <= 1e-4 * np.abs(w).max()
        assert np.array_equal(g, a)
