"""Small batches, whose whole forest one block builds (up to 2,048 bodies in all)
and sums (up to 4,096): several roots, a box per system, system edges inside a
warp and at a block's tile edge.  Every system steps bit for bit as it does alone."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [10, 20])
@pytest.mark.parametrize("counts", [[2, 2, 33, 700], [31, 32, 33, 64, 2], [1023, 2, 1023], [1024, 1024], [2] * 64,
                                    [1025, 1024], [1000, 1500, 777], [2047, 2, 2047], [4000, 96], [4000, 97]])
def test_small_batch_equals_systems_alone(torch_cuda, engine, counts, bits):
    off = np.concatenate([[0], np.cumsum(counts)])
    pos, vel = np.empty((off[-1], 4), np.float32), np.empty((off[-1], 3), np.float32)
    for k, n in enumerate(counts):
        sl = slice(off[k], off[k + 1])
        pos[sl], vel[sl] = engine.plummer(n, seed=70 + k)
        pos[sl, :3] *= np.float32(1 + 0.5 * (k % 5))  # extents of their own
        pos[sl, :3] += np.float32(3 * (k % 7))
        if n > 100:  # bodies in one place
            pos[off[k] + 5:off[k] + 12, :3] = pos[off[k] + 4, :3]
    prm = engine.Params(bits_per_axis=bits, theta=0.5, eps=0.01, dt=1e-3)
    with engine.Simulation(0, prm, counts=counts) as b:
        b.load(pos, vel)
        acc = b.accelerations()
        inter, nodes = b.stats()["interactions"], b.stats()["node_count"]
        b.step(3)
        bp, bv = b.store()
    total = trees = 0
    for k, n in enumerate(counts):
        sl = slice(off[k], off[k + 1])
        with engine.Simulation(n, prm) as s:
            s.load(pos[sl], vel[sl])
            a = s.accelerations()
            total += s.stats()["interactions"]
            trees += s.stats()["node_count"]
            s.step(3)
            sp, sv = s.store()
        assert np.array_equal(acc[sl], a), f"system {k}: forces differ"
        assert np.array_equal(bp[sl], sp) and np.array_equal(bv[sl], sv), f"system {k}: state differs"
    assert inter == total and nodes == trees
