"""The stages of the staged collide-and-stream kernels are refilled only after they have been read: the same state
stepped again and again gives the same bits.  Rows that the linear tiles take and rows that the row tiles take; the
walls' cells keep the shared-memory pipe busy with global loads, and steps follow each other so closely that refills
come from L2.  (Without the proxy fence before a stage's release about one warp in 3 x 10^8 read the next tile's values:
in FP32 on 313 x 79 x 89 one step in 5,000.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bib = pytest.importorskip("biblbm_gb300")


@pytest.mark.parametrize("storage,nx,repeats", [("f32", 313, 100), ("f32", 312, 20), ("f16", 313, 20), ("f16", 320, 20), ("f64", 128, 4)])
def test_repeated_steps_give_the_same_bits(storage, nx, repeats):
    ny, nz = 79, 89
    rng = np.random.default_rng(5)
    u0 = rng.uniform(-0.02, 0.02, (3, nz, ny, nx))
    ctx = bib.Context(0)
    try:
        lat = ctx.add_domain(nx, ny, nz, storage=storage, periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb", omega=1.1,
                             body_force=(1e-6, 2e-6, -1e-6))
        want = None
        for _ in range(repeats):
            lat.initialize_at_equilibrium(None, u0)
            lat.collide_and_stream(200)
            got = lat.compute_velocity()
            if want is None:
                want = got
            assert np.array_equal(got, want)
        lat.check_health()
    finally:
        ctx.close()
