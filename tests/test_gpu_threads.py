"""Handles in several host threads at once (distinct handles are independent):
rooms whose on-chip solves share a kernel and differ in the shared memory it
needs, by turns in every thread, give what they give alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# per form a room with a large plane (or row) and one with a small one
FORMS = [((2, 60, 60), (90, 8, 10)), ((4, 60, 60), (180, 8, 10)), ((5, 70, 71), (310, 8, 10)), ((12, 61, 66), (480, 10, 10)),
         ((6, 120, 100), (150, 120, 4))]


@pytest.mark.parametrize("grids", FORMS)
def test_threads_solve_side_by_side(grids):
    import torch
    from ffrb import capi
    from ffrb.scene import Patch, add_outflow, empty_room
    work = []
    for g in grids * 2:
        room = empty_room(*g, 4.0, 3.0, 2.5)
        add_outflow(room, Patch(0, 1, 0, g[1] - 1, 0, g[2] - 1))
        h = capi.PoissonHandle(room, 2, 1e-13)
        rhs = torch.as_tensor(np.random.default_rng(3).standard_normal(room.n_cells), device="cuda")
        x = torch.empty_like(rhs)
        torch.cuda.synchronize()
        h.solve_dev(rhs.data_ptr(), x.data_ptr())
        work.append((h, rhs, x, x.clone()))
    torch.cuda.synchronize()
    errors = []

    def loop(h, rhs, x):
        try:
            for _ in range(2000):
                h.solve_dev(rhs.data_ptr(), x.data_ptr())
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=loop, args=w[:3]) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for h, _, x, alone in work:
        assert torch.equal(x, alone)
        h.close()
