"""Box and keys of a small system in one block (up to 8,192 bodies), around the
edges of its threads: keys and order are the oracle's, the root's FP64
sums are numpy's to rounding (n terms, at most n 2^-53 of the sum of their
magnitudes in either order), and its last body is looked at as closely as the
others."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev_to_host

pytestmark = pytest.mark.gpu

SIZES = [2, 33, 1024, 1025, 4096, 4097, 7169, 8192, 8193]


@pytest.mark.parametrize("bits", [10, 21])
@pytest.mark.parametrize("n", SIZES)
def test_small_box_and_keys(torch_cuda, engine, oracle, n, bits):
    p, v = engine.plummer(n, seed=n + bits)
    ref = oracle.pipeline(p, v, bits)
    with engine.Simulation(n, engine.Params(bits_per_axis=bits, eps=0.01)) as sim:
        sim.load(p, v)
        sim.accelerations()
        root, ts = sim.root_f64(), sim.tree()
        assert np.array_equal(dev_to_host(ts.mortonIn, (n,), np.uint64), ref["keys"])
        assert np.array_equal(dev_to_host(ts.indexOut, (n,), np.uint32), ref["perm"])
    q = p.astype(np.float64)
    assert np.array_equal(root["min"], q[:, :3].min(0)) and np.array_equal(root["max"], q[:, :3].max(0))
    rounding = 2 * n * 2.0**-53
    mass = q[:, 3].sum()
    assert abs(root["mass"] - mass) <= rounding * mass
    mx = q[:, 3:] * q[:, :3]
    assert np.all(np.abs(root["com"] - mx.sum(0) / mass) <= 2 * rounding * np.abs(mx).sum(0) / mass)


@pytest.mark.parametrize("n", [33, 1025, 4096, 8192])
def test_small_box_reports_the_last_body(torch_cuda, engine, n):
    p, v = engine.plummer(n, seed=1)
    p[-1, 2] = np.nan
    with engine.Simulation(n, engine.Params(eps=0.01)) as sim:
        sim.load(p, v)
        with pytest.raises(engine.BHError) as e:
            sim.accelerations()
            sim.stats()
        assert "NONFINITE" in e.value.name
