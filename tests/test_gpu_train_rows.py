"""Every row of a training epoch counts, once and in its own batch.

The network here has small whole numbers for weights and inputs, so activations
and errors are exact in BF16 and FP32 whatever the order of a sum: no rounding
flips between the kernels and the oracle, and what is left is the FP32 summation
of the gradients (some 1e-6 of their norm at 65,539 rows; one lost row is 4e-3).
With a learning rate of 0 every batch sees the same weights, and the moments
collect all batches' gradients.  After real steps weights are rounded to BF16
anew in every batch and an epoch amplifies the order of its sums (two runs of
float atomics end 1e-3 apart after 256 batches), so that equality is only asked
of one batch."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2
from oracle import mlp as M

pytestmark = pytest.mark.gpu

TOL = 1e-5
CASES = [(16, 16), (17, 16), (100, 33), (1000, 250), (4096, 4096), (8193, 4096), (5000, 20000), (8200, 8192),
         (9000, 9000), (12345, 777), (20000, 8193), (65539, 8192), (65539, 40000), (65539, 65539)]


def _whole_numbers(rows):
    rng = np.random.default_rng(rows)
    p = np.zeros(M.TOTAL, np.float32)
    w = M.blocks(p)
    w["W1"][:] = rng.integers(-1, 2, (8, 32))
    w["b1"][:] = rng.integers(-1, 2, 32)
    w["W2"][:] = rng.integers(-1, 2, (32, 32)) * (rng.random((32, 32)) < 0.4)
    w["b2"][:] = rng.integers(-1, 2, 32)
    w["W3"][:] = rng.integers(-1, 2, 32)
    w["b3"][:] = 1
    w["inv_std"][:] = 1
    X = rng.integers(-2, 3, (rows, 8)).astype(np.float32)
    y, _ = M.forward_bf16(p, X)
    return p, X, y


def _epoch(torch, p, X, Y, batch, lr, v0=0.0):
    from cudagravitydemo_b200 import learned
    tr = learned.Trainer(p)
    tr.v.fill_(v0)
    tr.step.value = 500
    mse = tr.epoch(torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda(), batch, lr)
    return tr, mse


def _moments(p, X, Y, batch, v0=0.0):
    m, v, se, g = np.zeros(M.TRAINED), np.full(M.TRAINED, v0), 0.0, None
    for r in range(0, len(Y), batch):
        g, lo = M.grad_bf16(p, X[r:r + batch], Y[r:r + batch])
        m, v, se = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g, se + lo
    return m, v, se, g


@pytest.mark.parametrize("rows,batch", CASES)
def test_all_batches_of_an_epoch(torch_cuda, engine, rows, batch):
    p, X, y = _whole_numbers(rows)
    Y = (y + np.random.default_rng(1).integers(-3, 4, rows)).astype(np.float32)
    tr, mse = _epoch(torch_cuda, p, X, Y, batch, 0.0)
    m, v, se, g = _moments(p, X, Y, batch)
    assert tr.step.value == 500 + -(-rows // batch)
    assert np.array_equal(tr.params(), p)
    assert mse * rows == pytest.approx(se, rel=1e-6)
    assert rel_l2(tr.m.cpu().numpy(), m) < TOL
    assert rel_l2(tr.v.cpu().numpy(), v) < 2 * TOL
    assert rel_l2(tr.grad.cpu().numpy(), g) < TOL


@pytest.mark.parametrize("rows,batch", CASES)
def test_one_wrong_row_is_seen(torch_cuda, engine, rows, batch):
    torch = torch_cuda
    p, X, y = _whole_numbers(rows)
    last = (rows - 1) // batch * batch  # first row of the last batch
    at = {0, 15, 16, 4095, 4096, batch - 17, batch - 16, batch - 1, batch, last, last + 15, rows - 17, rows - 1,
          37887, 37888, 37903}
    for r in sorted(a for a in at if 0 <= a < rows):
        Y = y.copy()
        Y[r] += 3
        tr, mse = _epoch(torch, p, X, Y, batch, 0.0)
        assert mse * rows == pytest.approx(9.0, rel=1e-6), r
        own = slice(r // batch * batch, r // batch * batch + batch)
        g, _ = M.grad_bf16(p, X[own], Y[own])
        later = (rows - 1) // batch - r // batch  # batches after the row's own
        assert rel_l2(tr.m.cpu().numpy(), 0.1 * 0.9 ** later * g) < TOL, r
        if later == 0:
            assert rel_l2(tr.grad.cpu().numpy(), g) < TOL, r


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 63, 65, 1000, 37888, 37889, 40000, 65539])
def test_gradient_of_all_rows(torch_cuda, engine, rows):
    torch = torch_cuda
    from cudagravitydemo_b200 import learned
    p, X, y = _whole_numbers(rows)
    Y = (y + np.random.default_rng(1).integers(1, 4, rows)).astype(np.float32)
    g, loss = learned.loss_grad(*(torch.from_numpy(a).cuda() for a in (p, X, Y)))
    want, se = M.grad_bf16(p, X, Y)
    assert float(loss) == pytest.approx(se, rel=1e-6)
    assert rel_l2(g.cpu().numpy(), want) < TOL


@pytest.mark.parametrize("rows", [16, 17, 1000, 4096, 8192, 8193, 40000, 65539])
def test_a_step_moves_the_weights(torch_cuda, engine, rows):
    p, X, y = _whole_numbers(rows)
    Y = (y + np.random.default_rng(1).integers(-3, 4, rows)).astype(np.float32)
    lr = 1e-2
    tr, _ = _epoch(torch_cuda, p, X, Y, rows, lr, v0=1e-2)
    m, v, _, _ = _moments(p, X, Y, rows, v0=1e-2)
    moved = -lr * (m / (1 - 0.9 ** 501)) / (np.sqrt(v / (1 - 0.999 ** 501)) + 1e-8)
    got = tr.params().astype(np.float64) - p
    # a weight of up to 1 is rounded to 2^-24 (steps are up to 1e-2)
    assert np.linalg.norm(got[:M.TRAINED] - moved) < TOL * np.linalg.norm(moved) + 2.0 ** -24 * np.sqrt(M.TRAINED)
    assert np.array_equal(tr.params()[M.TRAINED:], p[M.TRAINED:])
