"""Every form of the multigrid solve against the whole-GPU one, whose V-cycle runs
in global memory (smooth_color, restrict_level, block_vcycle): the on-chip V-cycle
of one cluster and of the split solve, and the split solve whose coarse levels do
not fit a cluster's shared memory (8 x 180 x 180: 4 planes of 90 x 90).

The forms apply the same preconditioner cell update for cell update and differ in
the order of the FP64 dot products only, so their iteration counts differ by one
at most; a fault in a coarse level that both on-chip forms share would cost
iterations here.  All stop at 1e-9 (relative residual), which leaves the fields
within 1e-6 of each other."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

ROOMS = [((48, 40, 27), 1.0), ((34, 36, 25), 1.0), ((17, 70, 9), 1.0), ((90, 24, 64), 1.0), ((9, 30, 31), 1.0),
         ((50, 36, 25), 1.02), ((110, 70, 51), 1.0), ((12, 11, 10), 1.0), ((8, 180, 180), 1.0), ((96, 80, 41), 1.0)]


@pytest.mark.parametrize("grid,stretch", ROOMS)
def test_forms_agree_with_the_whole_gpu_solve(grid, stretch):
    from ffrb import capi, workloads
    from ffrb.params import params_from_scene
    from ffrb.scene import build_room
    cfg, _ = workloads.large_thermal(grid)
    cfg.room.stretch = stretch
    cfg.solver.poisson_tol = 1e-9
    cfg.solver.dt = workloads.room_dt(cfg)
    room, params = build_room(cfg), params_from_scene(cfg)

    def run(cluster, split):
        h = capi.FluidHandle(room, params)
        if cluster:
            h.set_cluster(cluster)
        else:
            h.set_split(split)
        recs = h.advance(3)
        assert all(r["flags"] == 0 for r in recs)
        out = [r["cg_iterations"] for r in recs], {k: h.get(k) for k in "uvwp"}
        h.close()
        return out

    want_its, want = run(0, 0)
    for form in ((0, 1), (1, None), (5, None), (16, None)):
        its, got = run(*form)
        assert max(abs(a - b) for a, b in zip(its, want_its)) <= 1, (form, its, want_its)
        for k in "uvwp":
            assert rel_err(got[k], want[k]) <= 1e-6, (form, k)
    assert np.isfinite(want["p"]).all()
