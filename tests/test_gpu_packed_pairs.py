"""FP16 collide-and-stream by packed pairs of cells: the shortest rows, walls that move, two viscosities
within a pair, nodes that are not collided beside ones that are, against the row kernel's one cell at a
time.  Both work in FP32 from the same values and round once, so that after one step they differ by at
most one unit in the last place of FP16 of the largest value (2^-10 of it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


WALLS = {"none": dict(), "channel": dict(periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb",
                                         wall_u=[[0.02, 0, 0.01], [-0.01, 0, 0], [0, 0.01, 0], [0.01, 0, 0]]),
         "fd": dict(periodic=(1, 0, 1), wall_y="fd_velocity", wall_u=[[-0.02, 0, 0], [0.02, 0, 0], [0, 0, 0], [0, 0, 0]])}


@pytest.mark.parametrize("typed", [False, True])
@pytest.mark.parametrize("walls", ["none", "channel", "fd"])
@pytest.mark.parametrize("collision", ["bgk_guo_vof", "bgk", "trt"])
@pytest.mark.parametrize("dims", [(8, 5, 4), (40, 12, 6), (512, 4, 4)])
def test_pairs_match_single_cells(ctx, dims, collision, walls, typed):
    nx, ny, nz = dims
    rng = np.random.default_rng(11)
    rho = 1 + rng.uniform(-0.02, 0.02, (nz, ny, nx))
    u = rng.uniform(-0.05, 0.05, (3, nz, ny, nx))
    F = rng.uniform(-1e-3, 1e-3, (3, nz, ny, nx))
    types = rng.integers(0, 3, (nz, ny, nx)).astype(np.uint8) * (rng.uniform(size=(nz, ny, nx)) < 0.3)
    out = []
    for kernel in ("staged", "rows"):
        lat = ctx.add_domain(nx, ny, nz, omega=1.3, omega_inner=0.8, storage="f16", collision=collision,
                             use_phase=collision == "bgk_guo_vof", **WALLS[walls])
        if typed:
            lat.set_cell_types(types.astype(np.uint8))
        lat.set_tuning(kernel=kernel)
        lat.initialize_at_equilibrium(rho, u)
        lat.set_external_force(F)
        if collision == "bgk_guo_vof":
            lat.set_phase((np.random.default_rng(5).uniform(size=(nz, ny, nx)) < 0.5).astype(np.uint8))
        lat.collide_and_stream(1)
        out.append(lat.receive())
    assert np.isfinite(out[0]).all()
    assert np.abs(out[0] - out[1]).max() <= 2.0 ** -10 * np.abs(out[1]).max()
