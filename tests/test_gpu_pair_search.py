"""Particle-particle forces by the warp-per-vertex search in boxes that strain it: a long periodic axis
(FP32 pre-test at large coordinates), pairs across periodic faces, walled axes, and two potentials
with different cutoffs.  FP64 against the oracle's all-pairs sum to 1e-12 of the largest component
(the order of a vertex's sum, fused multiply-adds and exp)."""
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


@pytest.mark.parametrize("dims,periodic,at", [((1500, 12, 12), (1, 1, 1), (1499.2, 11.5, 5.5)), ((9, 9, 9), (1, 1, 1), (0.1, 8.7, 4.0)),
                                              ((11, 40, 12), (1, 0, 1), (10.6, 34.0, 11.9)), ((16, 14, 70), (1, 0, 0), (15.8, 7.0, 62.0))])
@pytest.mark.parametrize("spread", ["atomic", "deterministic"])
def test_pair_forces_match_all_pairs(ctx, dims, periodic, at, spread):
    rng = np.random.default_rng(5)
    xyz, tri = meshes.icosphere(2, 1.9)
    gap = 0.5
    at = np.array(at)
    pos = [meshes.place(xyz, meshes.random_rotation(rng), at + s * (3.8 + gap) * np.eye(3)[a]) for a, s in ((0, 0), (0, 1), (1, -1))]
    prm = bib.membrane_params(G=1e-6, C=1.0)
    walls = {"wall_y": "none" if periodic[1] else "halfway_bb", "wall_z": "none" if periodic[2] else "halfway_bb"}
    pots = [("spring", 0.7, 0.0, 2e-3), ("morse", 1.0, 1.5, 1e-4)]
    L = O.lattice(dims, periodic, "bgk_guo_vof", 1.0, 1.0, **walls)
    S = O.System(L, "roma", -1.0)
    sid = S.add_shape(xyz, tri)
    lat = ctx.add_domain(*dims, periodic=periodic, omega=1.0, **walls)
    shapes = bib.ParticleShapeLibrary(ctx)
    gsid = shapes.store_mesh(xyz, tri, "c")
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, spread=spread)
    for p in pos:
        S.add_particle(sid, "capsule_skalak", prm, p)
        fsi.add_particle(gsid, "capsule_skalak", prm, p)
    for kind, r0, beta, k in pots:
        S.add_pp_interaction(O.potential(kind, r0, beta, k))
        fsi.add_pp_force(bib.SpringPotential(r0, k) if kind == "spring" else bib.MorsePotential(r0, beta, k))
    for _ in range(2):  # the second step searches with the buckets of the first cleared
        S.step(1)
        fsi.step(1)
    want = np.concatenate([S.particle(i)["force"] for i in range(3)])
    got = np.concatenate([fsi.get_particle(i)["force"] for i in range(3)])
    assert np.abs(want).max() > 1e-5
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
