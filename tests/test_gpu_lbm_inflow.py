"""INFLOW cells that no fan covers: the reference neither collides nor replaces
their populations (LBMSolver.cpp's inflow and collision loops both pass them by),
so what streams into such a cell is what the next step streams out, also where a
population is not finite or a zero is negative.

Narrow storages are compared with the FP64 storage, which takes the cells one by
one: the same populations finite, and those within the rounding of one store."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,tol", [("fp32", 2e-7), ("fp16", 1e-3)])
@pytest.mark.parametrize("grid", [(12, 10, 8), (11, 9, 7), (11, 10, 7)])
def test_fanless_inflow_keeps_what_arrives(grid, storage, tol):
    from ffrb import capi
    from ffrb.scene import empty_room
    room = empty_room(*grid, 0.1 * grid[0], 0.1 * grid[1], 0.1 * grid[2])
    types = room.cell_type.reshape(grid)
    cells = [(5, 4, 3), (5, 5, 4), (0, 4, 3), (3, 4, 4), (3, 4, 5)]     # both places of a pair, a wall, a whole pair
    for c in cells:
        types[c] = 2
    tau, dt = 0.8, 1e-3
    got = {}
    for s in ("fp64", storage):
        h = capi.LbmHandle(room, tau, 100, 1e-30, dt, s)
        f, step = h.get_populations()
        g = f.reshape((19,) + grid)
        g += 0.01 * np.random.default_rng(2).standard_normal(g.shape) * g
        # a value that is not finite streams into the first two cells (from every neighbour, in one direction each)
        for q in range(1, 19):
            for c in cells[:2]:
                g[q, c[0] - 1:c[0] + 2, c[1] - 1:c[1] + 2, c[2] - 1:c[2] + 2] = np.inf if q % 5 == 1 else g[q, c[0], c[1], c[2]]
        h.set_populations(f, step)
        h.advance(1)
        got[s] = h.get_populations()[0].reshape((19,) + grid)
        h.close()
    for c in cells:
        want, have = (got[s][(slice(None),) + c] for s in ("fp64", storage))
        assert np.array_equal(np.isinf(want), np.isinf(have)) and not np.isnan(have).any(), (c, have)
        ok = np.isfinite(want)
        assert np.abs(have[ok] - want[ok]).max() <= tol, c
    assert np.isinf(got["fp64"][(slice(None),) + cells[0]]).any()
