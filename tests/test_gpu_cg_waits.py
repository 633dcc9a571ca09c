"""The bounded waits of the on-chip CG: one block of the solve stays away from a
reduction, so every other block's wait runs out (under a limit of 50 ms).  The
call reports it, every copy between the blocks has arrived before a block left
(also those of a halo, pushed in the odd reductions), and the handle then solves
as before, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one to eight cells per thread in a cluster, then the chunked grid
ROOMS = [(16, 16, 16), (25, 20, 30), (33, 32, 24), (40, 39, 32), (50, 40, 40)]


@pytest.mark.parametrize("grid", ROOMS)
def test_waits_run_out(grid):
    from ffrb import capi
    from ffrb.scene import Patch, add_outflow, empty_room
    room = empty_room(*grid, 4.0, 3.0, 2.5)
    add_outflow(room, Patch(0, 1, 0, grid[1] - 1, 0, grid[2] - 1))
    rhs = np.random.default_rng(5).standard_normal(room.n_cells)
    h = capi.PoissonHandle(room, 12, 1e-13)
    before = h.solve(rhs)
    capi.set_device_wait_limit(0.05)
    try:
        for reduction in (1, 2, 3, 4, 5, 24, 25):
            status, lost, ms = h.selftest_wait(rhs, reduction)
            assert status == capi.FFR_ETIMEDOUT and lost == 0, (reduction, status, lost)
            assert 40.0 <= ms <= 3000.0, (reduction, ms)
        # (12 iterations: 25 reductions in a cluster, 26 in the grid)
        assert h.selftest_wait(rhs, 40)[:2] == (capi.FFR_OK, 0)
    finally:
        capi.set_device_wait_limit(0.0)
    after = h.solve(rhs)
    assert np.array_equal(before[0], after[0]) and before[1:] == after[1:]
    h.close()
