"""An epoch of training step by step against the oracle's BF16 gradient and a
plain Adam, at batches around a warp's 16 rows, a block's and a cluster's, with
ragged last batches, and on either side of the one-launch epoch's limit.

The gradients differ from the oracle's by FP32 summation order (1e-7 relative);
Adam's second moments start at 1e-2, far above the gradients' squares, so a step
is a smooth function of its gradient and the parameters agree to a few 1e-6 of
the distance they moved."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2
from oracle import mlp as M

pytestmark = pytest.mark.gpu

CASES = [(16, 16), (17, 16), (100, 33), (1000, 250), (4096, 4096), (8193, 4096), (5000, 20000), (8200, 8192),
         (20000, 8193), (9000, 9000)]


@pytest.mark.parametrize("rows,batch", CASES)
def test_epoch_matches_stepwise_adam(torch_cuda, engine, rows, batch):
    torch = torch_cuda
    from cudagravitydemo_b200 import learned
    rng = np.random.default_rng(rows)
    X = rng.normal(0, 1.5, (rows, 8)).astype(np.float32)
    Y = rng.normal(-2, 0.5, rows).astype(np.float32)
    p0 = learned.init_params(X.mean(0), X.std(0) + 1e-3, 3)
    tr = learned.Trainer(p0)
    tr.v.fill_(1e-2)
    tr.step.value = 500
    lr = 1e-2
    mse = tr.epoch(torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda(), batch, lr)

    p = p0.astype(np.float64)
    m, v = np.zeros(M.TRAINED), np.full(M.TRAINED, 1e-2)
    se, t, g = 0.0, 500, None
    for r in range(0, rows, batch):
        g, lo = M.grad_bf16(p.astype(np.float32), X[r:r + batch], Y[r:r + batch])
        se += lo
        t += 1
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p[:M.TRAINED] -= lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    assert tr.step.value == t
    assert mse == pytest.approx(se / rows, rel=1e-3)
    got = tr.params()
    moved = p[:M.TRAINED] - p0[:M.TRAINED]
    assert rel_l2(got[:M.TRAINED] - p0[:M.TRAINED], moved) < 2e-3  # the oracle test's gradient tolerance
    assert np.array_equal(got[M.TRAINED:], p0[M.TRAINED:])
    assert rel_l2(tr.m.cpu().numpy(), m) < 2e-3 and rel_l2(tr.v.cpu().numpy(), v) < 2e-3
    assert rel_l2(tr.grad.cpu().numpy(), g) < 2e-3
