"""Area, volume and centre of FP32 particles on both sides of the triangle count from which several CTAs share a
particle, against the oracle's sums: 2e-6 of the area and volume (triangles in FP32 relative to the centre, a few
roundings of 6e-8 each, summed per thread in FP32), 2e-6 of the radius for the centre."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")
from biblbm_gb300 import meshes  # noqa: E402


def ring_sphere(rings, segments, r):
    """A sphere of rings, 2 (rings - 1) segments triangles."""
    t = np.pi * np.arange(1, rings) / rings
    a = 2 * np.pi * np.arange(segments) / segments
    body = np.stack([np.sin(t)[:, None] * np.cos(a), np.sin(t)[:, None] * np.sin(a), np.cos(t)[:, None] + 0 * a], -1).reshape(-1, 3)
    xyz = r * np.concatenate([[[0, 0, 1.0]], body, [[0, 0, -1.0]]])
    at = lambda i, j: 1 + i * segments + j % segments  # noqa: E731
    tri = [[0, at(0, j), at(0, j + 1)] for j in range(segments)]
    for i in range(rings - 2):
        for j in range(segments):
            tri += [[at(i, j), at(i + 1, j), at(i, j + 1)], [at(i, j + 1), at(i + 1, j), at(i + 1, j + 1)]]
    tri += [[len(xyz) - 1, at(rings - 2, j + 1), at(rings - 2, j)] for j in range(segments)]
    return xyz, np.array(tri)


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("rings,segments", [(17, 63), (17, 64), (25, 60), (41, 66)])
@pytest.mark.parametrize("cells", [1, 3])
def test_sums_match_oracle(ctx, rings, segments, cells):
    xyz, tri = ring_sphere(rings, segments, 8.0)
    lat = ctx.add_domain(64, 40, 40, omega=1.0, storage="f32", body_force=(1e-5, 0, 0))
    shapes = bib.ParticleShapeLibrary(ctx)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes)
    sid = shapes.store_mesh(xyz, tri, "s")
    for k in range(cells):
        fsi.add_particle(sid, "capsule_skalak", bib.membrane_params(G=1e-4, C=1.0),
                         xyz * np.array([1.1, 0.95, 1.0]) + np.array([62.0 + 18 * k, 19.3, 20.4]))
    fsi.step(2)
    pos, stats = fsi.download()  # the device's sums
    for p, got in zip(pos.reshape(cells, -1, 3), stats):
        want = O.particle_update(p, tri)
        assert abs(got[0] - want[0]) <= 2e-6 * want[0] and abs(got[1] - want[1]) <= 2e-6 * want[1]
        assert np.abs(got[2:] - want[2:]).max() <= 2e-6 * 8.0
