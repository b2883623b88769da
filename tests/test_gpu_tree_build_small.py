"""Count, level table and nodes of a small tree in one block (up to 2,048
bodies), around the edges of its threads and of the node capacity: every node
bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev_to_host, node_fields_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [10, 21])
@pytest.mark.parametrize("n", [2, 31, 33, 1024, 1025, 2047, 2048, 2049])
def test_small_build_matches_oracle(torch_cuda, engine, oracle, n, bits):
    p, v = engine.plummer(n, seed=n)
    ref = oracle.pipeline(p, v, bits)
    with engine.Simulation(n, engine.Params(bits_per_axis=bits, eps=0.01, export_nodes=True)) as sim:
        sim.load(p, v)
        sim.accelerations()
        st = sim.stats()
        nodes = dev_to_host(sim.tree().nodes, (st["node_count"],), engine.NODE_DTYPE)
    assert st["node_count"] == ref["count"] and st["deepest_level"] == ref["deepest"]
    assert node_fields_equal(nodes, ref["nodes"]) == []


@pytest.mark.parametrize("n", [200, 2048, 2050])
def test_too_many_nodes_are_reported(torch_cuda, engine, n):
    rng = np.random.default_rng(n)
    p = np.empty((n, 4), np.float32)
    p[0::2, :3] = rng.uniform(0.25, 1, (n // 2, 3))
    p[1::2, :3] = np.nextafter(p[0::2, :3], np.float32(2))  # a chain of some 17 nodes above each pair: over 8 a body
    p[:, 3] = 1.0 / n
    with engine.Simulation(n, engine.Params(eps=0.01)) as sim:
        sim.load(p, np.zeros((n, 3), np.float32))
        with pytest.raises(engine.BHError) as e:
            sim.accelerations()
            sim.stats()
        assert e.value.name == "BH_ERR_TREE_OVERFLOW"
