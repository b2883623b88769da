"""The walk at the edges of its batches: groups that do not fill a block, a
last group of one body, 32- and 64-body groups, lists and buffers that end on
either side of a multiple of 32, and a traversal stack that spills.  The oracle
takes one node at a time, so equal interaction counts mean equal decisions."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5  # the tolerance of the walk's parity tests (rsqrt and summation order)

SIZES = [2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 257, 961, 4095, 4097, 18945]


@pytest.mark.parametrize("stack", [0, 128])
@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("n", SIZES)
def test_walk_edges_match_oracle(torch_cuda, engine, oracle, n, width, stack):
    p, v = engine.plummer(n, seed=n)
    ref = oracle.pipeline(p, v, 21)
    for theta in (0.25, 0.7):
        with engine.Simulation(n, engine.Params(theta=theta, eps=0.01, dt=1e-3, group_width=width)) as sim:
            if stack:
                sim.set_walk_stack(stack)
            sim.load(p, v)
            acc = sim.accelerations()
            st = sim.stats()
        want, inter = oracle.walk(ref["pos"], ref["nodes"], ref["ext_x"], 0.01, 1.0, theta, group=width)
        by_id = np.empty_like(want)
        by_id[ref["perm"]] = want
        assert st["interactions"] == inter
        assert rel_l2(acc, by_id) < FORCE_TOL
