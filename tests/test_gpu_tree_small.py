"""The octree at the edges of its one-block upward pass (4,096 bodies, 8,000
nodes): every node bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev_to_host, node_fields_equal

pytestmark = pytest.mark.gpu


def _pairs(n):
    """Close pairs: a chain of single children below each, six nodes a body."""
    rng = np.random.default_rng(n)
    p = np.empty((n, 4), np.float32)
    x = rng.uniform(0, 1, (n // 2, 3)).astype(np.float32)
    p[0::2, :3], p[1::2, :3] = x, x + np.float32(2e-5)
    p[:, 3] = rng.uniform(0.5, 1.5, n) / n
    p[5, 3] = 0.0  # a massless body
    return p, np.zeros((n, 3), np.float32)


@pytest.mark.parametrize("name,n", [("plummer", 3), ("plummer", 1023), ("plummer", 4095), ("plummer", 4096),
                                    ("plummer", 4097), ("pairs", 1000), ("pairs", 2000), ("pairs", 4096),
                                    ("pairs", 4098)])
def test_small_tree_matches_oracle(torch_cuda, engine, oracle, name, n):
    p, v = engine.plummer(n, seed=n) if name == "plummer" else _pairs(n)
    ref = oracle.pipeline(p, v, 21)
    if (name, n) == ("pairs", 2000):
        assert ref["count"] > 8000  # more nodes than the block holds
    with engine.Simulation(n, engine.Params(eps=0.01, export_nodes=True)) as sim:
        sim.load(p, v)
        sim.accelerations()
        st = sim.stats()
        nodes = dev_to_host(sim.tree().nodes, (st["node_count"],), engine.NODE_DTYPE)
    assert st["node_count"] == ref["count"] and st["deepest_level"] == ref["deepest"]
    assert node_fields_equal(nodes, ref["nodes"]) == []
