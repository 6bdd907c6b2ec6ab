"""Linear tiles (rows that no row tile takes) beside and before the membranes: steps with a capsule whose collision
only resets the previous force, steps with the sparse reset and consecutive (profiled) steps, against the direct
kernels; all pipeline depths; and the bounded waits.  Four steps from the same state: the kernels differ by a unit in
the last place of the populations (f-bar up to 0.004: FP16 1.9e-6, FP32 a few roundings, 4e-9) a step, which ten
populations of a velocity and the steps after it multiply by 10 at most for populations and by 100 for positions."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")
from biblbm_gb300 import _lib, meshes  # noqa: E402

DIMS = {"f16": (35, 33, 31), "f32": (83, 81, 79)}
U = [[-0.02, 0, 0], [0.02, 0, 0], [0, 0, 0], [0, 0, 0]]
WALLS = {"fd": dict(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=U),
         "channel": dict(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb", body_force=(1e-5, 0, 0))}


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


def capsule(ctx, storage, walls, **tuning):
    nx, ny, nz = DIMS[storage]
    lat = ctx.add_domain(nx, ny, nz, omega=1.1, storage=storage, **WALLS[walls])
    u0 = np.zeros((3, nz, ny, nx))
    u0[0] = (0.02 * (2 * np.arange(ny) / (ny - 1) - 1))[None, :, None]
    lat.initialize_at_equilibrium(None, u0)
    lat.set_tuning(**tuning)
    shapes = bib.ParticleShapeLibrary(ctx)
    xyz, tri = meshes.icosphere(2, 5.0)
    fsi = bib.ImmersedBoundaryDynamics3D(lat, shapes, spread="deterministic")
    pid = fsi.add_particle(shapes.store_mesh(xyz, tri, "c"), "capsule_skalak", bib.membrane_params(G=1e-3, C=1.0),
                           meshes.place(1.05 * xyz, None, (0.7, ny / 2 + 0.3, nz / 2 - 0.4)))
    return lat, fsi, pid


@pytest.mark.parametrize("walls", list(WALLS))
@pytest.mark.parametrize("storage", ["f16", "f32"])
def test_couplings_match_direct_kernels(ctx, storage, walls):
    ends = []
    for kernel, reset, profiled in (("rows", "auto", True), ("rows", "auto", False), ("auto", "auto", False), ("auto", "auto", True),
                                    ("auto", "sparse", False)):
        lat, fsi, pid = capsule(ctx, storage, walls, kernel=kernel, force_reset=reset)
        ctx.set_profiling(profiled)
        try:
            fsi.step(4)
        finally:
            ctx.set_profiling(False)
        lat.check_health()
        ends.append((lat.receive(), fsi.get_particle(pid)["pos"]))
    tol = {"f16": 2e-6, "f32": 4e-9}[storage]
    assert np.abs(ends[0][0]).max() < 0.01
    for f, pos in ends[1:]:
        assert np.abs(f - ends[0][0]).max() <= 40 * tol
        assert np.abs(pos - ends[0][1]).max() <= 400 * tol


@pytest.mark.parametrize("storage", ["f16", "f32"])
def test_depths_give_the_same_bits(ctx, storage):
    ends = []
    for stages in (0, 2, 3, 4):
        lat, fsi, pid = capsule(ctx, storage, "channel", stages=stages)
        fsi.step(3)
        lat.collide_and_stream(2)
        lat.check_health()
        ends.append((lat.receive(), fsi.get_particle(pid)["pos"]))
    for e in ends[1:]:
        assert np.array_equal(e[0], ends[0][0]) and np.array_equal(e[1], ends[0][1])


@pytest.mark.parametrize("storage,dims", [("f32", (83, 81, 79)), ("f32", (523, 33, 31)), ("f32", (514, 32, 33)), ("f16", (35, 33, 31)),
                                          ("f16", (34, 32, 31)), ("f16", (520, 9, 8)), ("f16", (1024, 6, 7))])
def test_withheld_tile_times_out(ctx, storage, dims):
    """Also says that these lattices take the linear tiles: the direct kernels wait for nothing."""
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    f0 = rng.uniform(-0.004, 0.004, (19, nz, ny, nx))
    lat = ctx.add_domain(nx, ny, nz, storage=storage, periodic=(1, 1, 1), omega=1.3)
    lat.set_tuning(wait_limit_us=2000, withhold_tile=7)
    lat.send(f0)
    t0 = time.perf_counter()
    lat.collide_and_stream(1)
    with pytest.raises(_lib.BibError) as e:
        lat.check_health()
    assert e.value.status == -5 and time.perf_counter() - t0 < 1.0  # BIB_ETIMEOUT
    lat.check_health()
    lat.set_tuning()
    lat.send(f0)
    lat.collide_and_stream(2)
    lat.check_health()
    ref = ctx.add_domain(nx, ny, nz, storage=storage, periodic=(1, 1, 1), omega=1.3)
    ref.send(f0)
    ref.collide_and_stream(2)
    assert np.array_equal(lat.receive(), ref.receive())


@pytest.mark.parametrize("storage", ["f16", "f32"])
def test_withheld_tile_beside_the_membranes(ctx, storage):
    lat, fsi, pid = capsule(ctx, storage, "channel", wait_limit_us=2000, withhold_tile=3)
    fsi.step(2)
    with pytest.raises(_lib.BibError) as e:
        lat.check_health()
    assert e.value.status == -5
    lat.set_tuning()
    fsi.step(2)  # steps again (the state of the failed step is not meaningful)
    assert np.isfinite(lat.receive()).all()
