"""Which form of a solve a room takes (no GPU needed): by its size on a device
that can place every cluster, and what it falls back to where one cannot be
placed.  csrc/forms.h is compiled into a small program; each line of its input is
a question."""
import os
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "forms.h"
int main(int argc, char **argv)
{
    if (argc == 3) {     // most blocks of the plain and of the on-chip kernel that can be placed
        const int most[2] = {std::atoi(argv[1]), std::atoi(argv[2])};
        const ffr::MidForm f = ffr::mid_form([&](bool onchip, int ctas) { return ctas <= most[onchip]; });
        std::printf("%d %d\n", f.ctas, (int)f.onchip);
        return 0;
    }
    int nx, ny, nz, smem, sms, pair, most;
    while (std::scanf("%d %d %d %d %d %d %d", &nx, &ny, &nz, &smem, &sms, &pair, &most) == 7)
        std::printf("%d\n", ffr::cg_form(nx, ny, nz, smem, sms, pair != 0, [=](int, int blocks) { return blocks <= most; }));
    return 0;
}
"""
SMEM, SMS = 232448 - 256, 148
CHUNKS, GRID = 0, -1


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    (d / "forms.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(PKG, "csrc"), str(d / "forms.cpp"),
                           "-o", str(d / "forms")])
    return str(d / "forms")


def ask(program, *question):
    return int(subprocess.run([program], input=" ".join(map(str, question)), text=True, capture_output=True,
                              check=True).stdout)


@pytest.mark.parametrize("grid,form", [((1, 1, 1), 1), ((8, 32, 32), 1), ((9, 32, 32), 2), ((16, 32, 32), 2), ((17, 32, 32), 4),
                                       ((32, 32, 32), 4), ((33, 32, 32), 8), ((64, 32, 32), 8), ((65, 32, 32), CHUNKS),
                                       ((128, 32, 32), CHUNKS), ((129, 32, 32), GRID), ((3, 200, 130), CHUNKS),
                                       ((2, 2, 30000), GRID), ((1, 80, 80), 1), ((1, 90, 90), GRID), ((1, 100, 92), CHUNKS)])
def test_by_size(program, grid, form):
    assert ask(program, *grid, SMEM, SMS, 1, 16) == form


@pytest.mark.parametrize("grid,most,form", [((25, 20, 12), 16, 1), ((25, 20, 12), 8, 2), ((25, 20, 12), 2, 8), ((25, 20, 12), 1, GRID),
                                            ((25, 20, 12), 0, GRID), ((41, 33, 19), 12, 8), ((41, 33, 19), 6, CHUNKS),
                                            ((64, 32, 32), 15, CHUNKS), ((64, 32, 32), 0, CHUNKS), ((5, 4, 3), 0, GRID)])
def test_where_a_cluster_cannot_be_placed(program, grid, most, form):
    assert ask(program, *grid, SMEM, SMS, 1, most) == form


def test_the_grid_form_needs_its_blocks_and_its_scratch(program):
    assert ask(program, 80, 64, 24, SMEM, SMS, 1, 16) == CHUNKS
    assert ask(program, 80, 64, 24, SMEM, 127, 1, 16) == GRID
    assert ask(program, 80, 64, 24, SMEM, SMS, 0, 16) == GRID
    assert ask(program, 80, 64, 24, 70000, SMS, 1, 16) == GRID


@pytest.mark.parametrize("plain,chip,want", [(16, 16, (16, 1)), (16, 15, (16, 0)), (15, 15, (8, 1)), (8, 0, (8, 0)), (7, 7, (1, 1)),
                                             (0, 0, (1, 0))])
def test_coarse_levels(program, plain, chip, want):
    out = subprocess.run([program, str(plain), str(chip)], text=True, capture_output=True, check=True).stdout
    assert tuple(map(int, out.split())) == want
