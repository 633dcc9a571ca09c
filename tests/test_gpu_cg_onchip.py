"""The on-chip CG (rooms of at most 131 072 cells) at the edges of its forms:
one to eight cells per thread in a cluster, the chunked grid, k_cg beyond.

Tolerance: both sides run the same CG in FP64 and differ in the order of the
dot products only, a relative 1e-15 per reduction; over the 30 iterations run
here that stays below 1e-10 of the solution's largest value unless the
iteration amplifies it, so 1e-9 (the bound of the solves in
test_gpu_poisson.py) with the same iteration count."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

SIZES = [(2, 1, 3), (3, 2, 2), (257, 1, 1), (16, 16, 1), (7, 39, 30), (8, 32, 32), (9, 32, 32), (64, 16, 16),
         (65, 16, 16), (32, 32, 32), (33, 32, 32), (64, 32, 32), (65, 32, 32), (3, 200, 130), (1100, 11, 10),
         (128, 32, 32), (129, 32, 32)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("stretch", [1.0, 1.01])
def test_onchip_cg_matches_oracle(size, stretch, oracle):
    from ffrb import capi
    from ffrb.scene import Patch, add_outflow, empty_room
    if stretch != 1.0 and min(size) == 1:
        pytest.skip("an axis of one cell has no stretched spacing")
    room = empty_room(*size, 4.0, 3.0, 2.5, stretch)
    rng = np.random.default_rng(list(size))
    if room.n_cells > 12:
        room.cell_type[rng.integers(0, room.n_cells, room.n_cells // 50 + 1)] = 1
    add_outflow(room, Patch(0, 1, 0, size[1] - 1, 0, size[2] - 1))     # (without it the system is singular)
    rhs = rng.standard_normal(room.n_cells)
    rhs[room.cell_type == 1] = 0.0
    h = capi.PoissonHandle(room, 30, 1e-13)
    x, res, it = h.solve(rhs)
    again, _, _ = h.solve(rhs)
    xo, reso, ito = oracle.cg_solve(room, rhs, 30, 1e-13)
    assert it == ito
    assert rel_err(x, xo) <= 1e-9 and abs(res - reso) <= 1e-9 * max(reso, 1.0)
    assert np.array_equal(x, again)
