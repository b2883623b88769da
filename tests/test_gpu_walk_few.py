"""Walks of few groups take a variant of the walk with more registers, up to 24
groups per SM: on either side of that line the interaction counts are the
oracle's, and a system walked alone (few groups) has the bits that it has in a
batch with a system of many groups."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5  # the tolerance of the walk's parity tests (rsqrt and summation order)


@pytest.mark.parametrize("over", [0, 1])
def test_walk_at_the_line_matches_oracle(torch_cuda, engine, oracle, over):
    n = 24 * 32 * torch_cuda.cuda.get_device_properties(0).multi_processor_count + over
    p, v = engine.plummer(n, seed=3)
    ref = oracle.pipeline(p, v, 21)
    with engine.Simulation(n, engine.Params(theta=0.7, eps=0.01, dt=1e-3)) as sim:
        sim.load(p, v)
        acc = sim.accelerations()
        st = sim.stats()
    want, inter = oracle.walk(ref["pos"], ref["nodes"], ref["ext_x"], 0.01, 1.0, 0.7, group=32)
    by_id = np.empty_like(want)
    by_id[ref["perm"]] = want
    assert st["interactions"] == inter
    assert rel_l2(acc, by_id) < FORCE_TOL


@pytest.mark.parametrize("leaf", [1, 16])
def test_few_and_many_groups_give_the_same_bits(torch_cuda, engine, leaf):
    counts = [33, 120001, 1000, 4097]
    bodies = [engine.plummer(n, seed=10 + k) for k, n in enumerate(counts)]
    prm = engine.Params(bits_per_axis=20, theta=0.5, eps=0.01, dt=1e-3, leaf_size=leaf)
    with engine.Simulation(0, prm, counts=counts) as batch:
        batch.load(np.concatenate([b[0] for b in bodies]), np.concatenate([b[1] for b in bodies]))
        acc = batch.accelerations()
        off = batch.system_offsets()
    for k, n in enumerate(counts):
        with engine.Simulation(n, prm) as sim:
            sim.load(*bodies[k])
            assert np.array_equal(acc[off[k]:off[k + 1]], sim.accelerations())
