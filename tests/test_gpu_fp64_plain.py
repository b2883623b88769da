"""The FP64 direct sum and pair potential against the plain formula where bodies,
masses and softenings are infinite, zero or nearly so."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _direct(torch, p, t, eps):
    from cudagravitydemo_b200 import accuracy
    return accuracy.direct_sum(torch.from_numpy(p).cuda(), torch.from_numpy(t).cuda(), eps, 1.0).cpu().numpy()


def _potential(engine, torch, p, eps):
    v = torch.zeros((len(p), 3), device="cuda")
    return engine.diagnostics(torch.from_numpy(p).cuda(), v, eps, 1.0)["potential"]


def _plain(p, eps):
    """Accelerations of all bodies and the potential, by the formula in 64 bits with its own infinities and NaN."""
    x, m = p[:, :3].astype(np.float64), p[:, 3].astype(np.float64)
    with np.errstate(all="ignore"):
        d = x[None] - x[:, None]
        ri = 1 / np.sqrt((d * d).sum(-1) + np.float64(eps) * np.float64(eps))
        acc = (((m * ri) * ri * ri)[..., None] * d).sum(1)
        w = m * ri
        np.fill_diagonal(w, 0.0)
        return acc, -0.5 * (m * w.sum(1)).sum()


def _edge(name, n):
    rng = np.random.default_rng(n)
    p = np.empty((n, 4), np.float32)
    p[:, :3] = rng.normal(0, 1, (n, 3))
    p[:, 3] = rng.uniform(0.1, 1, n) / n
    k = n - 2
    if name == "far":
        p[k, 0] = np.inf
    elif name == "far_below":
        p[k, 2] = -np.inf
    elif name == "two_far":
        p[k, 0], p[n - 1, 0] = np.inf, -np.inf
    elif name == "nan":
        p[k, 1] = np.nan
    elif name == "heavy":
        p[k, 3] = np.inf
    elif name == "heavy_and_massless":
        p[k, 3], p[0, 3] = np.inf, 0
    elif name == "coincident":
        p[k] = p[n - 1]
    elif name == "coincident_massless":
        p[k] = p[n - 1]
        p[k, 3] = 0
    return p


@pytest.mark.parametrize("name", ["plain", "far", "far_below", "two_far", "nan", "heavy", "heavy_and_massless",
                                  "coincident", "coincident_massless"])
@pytest.mark.parametrize("n", [2, 40, 700])
def test_infinite_zero_and_subnormal(torch_cuda, engine, n, name):
    p = _edge(name, n)
    t = np.arange(n, dtype=np.int32)
    # squares: 0, subnormal, tiny, ordinary, huge, infinite
    for eps in (0.0, 1e-160, 1e-150, 1e-60, 0.01, 1e100, 1e160, np.inf):
        acc, pot = _plain(p, eps)
        got = _direct(torch_cuda, p, t, eps)
        assert np.array_equal(np.isnan(got), np.isnan(acc)), (eps, "NaN")
        inf = np.isinf(acc)
        assert np.array_equal(got[inf], acc[inf]) and not np.isinf(got[~inf]).any(), (eps, "infinities")
        ok = np.isfinite(acc)
        assert np.allclose(got[ok], acc[ok], rtol=1e-10, atol=1e-10 * np.abs(acc[ok]).max(initial=0)), eps
        assert _potential(engine, torch_cuda, p, eps) == pytest.approx(pot, rel=1e-10, abs=0, nan_ok=True), eps
