"""Population transfers in the cell-major wire orders at the edges of the transfer tile (8 x-cells by
32 z-cells): the cell-major buffer is the transpose of the structure-of-arrays one to the bit, in both
directions, from page-locked and pageable memory."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
bib = pytest.importorskip("biblbm_gb300")

pytestmark = pytest.mark.gpu
CODE, PER = {"palabos": 1, "coprocessor": 2}, {"palabos": 23, "coprocessor": 19}


@pytest.fixture(scope="module")
def ctx():
    c = bib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("dims", [(3, 3, 3), (7, 3, 31), (8, 4, 32), (9, 3, 33), (17, 5, 70)])
@pytest.mark.parametrize("layout", ["palabos", "coprocessor"])
@pytest.mark.parametrize("storage", ["f64", "f16"])
def test_cell_major_order_is_the_transpose(ctx, dims, layout, storage):
    nx, ny, nz = dims
    lat = ctx.add_domain(nx, ny, nz, periodic=(1, 0, 0), wall_y="halfway_bb", wall_z="halfway_bb", storage=storage,
                         use_phase=True, omega_inner=1.0)
    rng = np.random.default_rng(sum(dims))
    # multiples of 2^-10 below 1/8: exact in FP16 storage scaled by 8192
    f = rng.integers(-100, 100, (19, nz, ny, nx)) / 1024.0
    force, phase = rng.integers(-8, 8, (3, nz, ny, nx)) / 64.0, rng.integers(0, 2, (nz, ny, nx)).astype(float)
    per = PER[layout]
    wire = np.concatenate([f, force, phase[None]])[:per].transpose(3, 2, 1, 0)
    for pinned in (True, False):
        buf = torch.empty((nx, ny, nz, per), dtype=torch.float64, pin_memory=pinned).numpy()
        buf[...] = wire
        ctx.check(ctx.lib.bib_lattice_send(ctx.h, lat.h, buf.ctypes.data, buf.nbytes, CODE[layout]))
        assert np.array_equal(lat.receive("soa"), f)
        buf[...] = np.nan
        ctx.check(ctx.lib.bib_lattice_receive(ctx.h, lat.h, buf.ctypes.data, buf.nbytes, CODE[layout]))
        assert np.array_equal(buf, wire)
        lat.send(np.zeros_like(f))
