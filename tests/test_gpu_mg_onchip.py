"""The on-chip V-cycle at the edges of its plans: cluster sizes, levels split
over blocks with a short last block, odd and even rows, thin rooms,
semi-coarsened and stretched grids, rooms too large for it on level 0.

The one-cluster solve and the one-kernel-per-pass solve apply the same
preconditioner cell update for cell update and differ in the order of the FP64
dot products only, so their iteration counts differ by one at most (where the
residual of an iteration lands beside the tolerance); both stop at 1e-9
(relative residual), which leaves the fields within 1e-6 of each other."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

ROOMS = [((48, 40, 27), 1.0), ((34, 36, 25), 1.0), ((80, 33, 18), 1.0), ((17, 70, 9), 1.0), ((90, 24, 64), 1.0),
         ((9, 30, 31), 1.0), ((50, 36, 25), 1.02), ((64, 64, 8), 1.0), ((110, 70, 51), 1.0), ((12, 11, 10), 1.0)]


@pytest.mark.parametrize("grid,stretch", ROOMS)
@pytest.mark.parametrize("ctas", [1, 5, 16])
def test_cluster_matches_split(grid, stretch, ctas):
    from ffrb import capi, workloads
    from ffrb.params import params_from_scene
    from ffrb.scene import build_room
    cfg, _ = workloads.large_thermal(grid)
    cfg.room.stretch = stretch
    cfg.solver.poisson_tol = 1e-9
    cfg.solver.dt = workloads.room_dt(cfg)
    room, params = build_room(cfg), params_from_scene(cfg)
    runs = []
    for cluster in (ctas, 0):
        h = capi.FluidHandle(room, params)
        if cluster:
            h.set_cluster(cluster)
        else:
            h.set_split(1)
        recs = h.advance(3)
        runs.append(([r["cg_iterations"] for r in recs], {k: h.get(k) for k in "uvwp"}))
        assert all(r["flags"] == 0 for r in recs)
        h.close()
    assert max(abs(a - b) for a, b in zip(runs[0][0], runs[1][0])) <= 1
    for k in "uvwp":
        assert rel_err(runs[0][1][k], runs[1][1][k]) <= 1e-6, k
