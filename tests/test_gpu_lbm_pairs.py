"""The lattice step where its variants change: even and odd rows and planes (one
or two loads per pair of cells), lattices whose last pair has one cell, rows of
one cell, re-mapped outflow cells at edges of openings, and both sides of the
sizes at which a cell pair replaces a cell (FP64 step, face velocities).

Bounds: those of the fixtures of the same length (FP64 sums in another order,
some 1e-13 after a few steps; FP32 and FP16 populations 2e-6 and 2e-3)."""
import numpy as np
import pytest

from oracle import new_fields

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-11, "fp32": 2e-6, "fp16": 2e-3}
SMALL = [(24, 20, 18), (23, 20, 15), (21, 17, 13), (30, 19, 1), (5, 3, 7), (40, 6, 2)]
LARGE = [((130, 120, 95), "fp64"), ((130, 120, 98), "fp64"), ((256, 196, 118), "fp32"), ((256, 196, 122), "fp32"),
         ((256, 196, 122), "fp64")]


def scene(grid):
    from ffrb.scene import (FanConfig, ObstacleConfig, OpeningConfig, RoomConfig, SceneConfig, build_room)
    lx, ly, lz = size = tuple(0.2 * n for n in grid)
    return build_room(SceneConfig(
        room=RoomConfig(size, grid), fans=[FanConfig((0.1, 0.5 * ly, 0.5 * lz), (0.0, 0.0), 2.0, 0.5, "west")],
        obstacles=[ObstacleConfig((0.4 * lx, 0.3 * ly, 0.0), (0.6 * lx, 0.6 * ly, 0.5 * lz), "box")],
        openings=[OpeningConfig("east", (0.7 * ly, 0.5 * lz), (0.6 * ly, 1.2 * lz), 20.0),
                  OpeningConfig("north", (0.8 * lx, 0.5 * lz), (0.5 * lx, 0.6 * lz), 20.0)]))


def check(oracle, grid, storage, steps):
    from ffrb import capi
    room = scene(grid)
    tau, dt = 0.8, 0.05 * room.dx / 2.0
    f, want = oracle.lbm_init(room, tau, dt), new_fields(room)
    oracle.lbm_run(room, tau, dt, 1e-30, f, want, steps)
    h = capi.LbmHandle(room, tau, 1000, 1e-30, dt, storage)
    h.advance(steps)
    speed = max(np.abs(want[k]).max() for k in "uvw")
    for k in "uvwp":
        err = np.abs(h.get(k) - want[k]).max() / (np.abs(want[k]).max() if k == "p" else speed)
        assert err <= TOL[storage], (k, err)
    h.close()


@pytest.mark.parametrize("grid", SMALL)
@pytest.mark.parametrize("storage", list(TOL))
def test_small(oracle, grid, storage):
    check(oracle, grid, storage, 8)


@pytest.mark.parametrize("grid,storage", LARGE)
def test_large(oracle, grid, storage):
    check(oracle, grid, storage, 2)
