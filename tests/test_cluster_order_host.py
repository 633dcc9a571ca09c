"""Order of a one-cluster solve's first accesses (no GPU needed): a block may
touch the shared memory of another one only once that block runs, so a cluster
barrier has to lie between a solve's start and its first reduction, which stores
into every block.  A missing one shows on a GPU by chance only, so the source is
what is looked at."""
import os
import re

from conftest import PKG

SRC = open(os.path.join(PKG, "csrc", "mgpcg.cu")).read()


def body(opening, text=SRC):
    """The braces' contents that follow `opening`."""
    at = text.index("{", text.index(opening))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i]
    raise AssertionError(opening)


def test_every_block_runs_before_the_first_reduction():
    group = body("struct ClusterGroup")
    init, ready = body("static void init()", group), body("static void ready()", group)
    assert "barrier.cluster.arrive" in init and "barrier.cluster.wait" in ready
    solve = body("pcg_body(const PCGArgs &A)")
    start, wait, first = (solve.index(s) for s in ("G::init()", "G::ready()", "allreduce<"))
    assert start < wait < first
    # on every path there, and with no other barrier of the cluster between arrival and wait
    between = solve[start:wait]
    assert not re.search(r"goto|return|G::sync|cluster", between)
    assert "cluster" not in body("void oc_setup", open(os.path.join(PKG, "csrc", "mgonchip.cuh")).read())
