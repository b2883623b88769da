"""The FP64 direct sum and pair potential against the plain formula: term by term
over the exponents that FP32 positions can give, with bodies, masses and
softenings that are infinite, zero or nearly so, and over several row tiles per
block of the potential."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# One term is 1/r^3 or 1/r from a rounded r^2, a series (relative error of what
# it leaves out 2^-55 and less) and at most five roundings: 8 of 2^-53 in all.
# Without the series' second term it would be off by up to 7e-12 and 1.4e-12.
TERM = 8 * 2.0 ** -53


def _direct(torch, p, t, eps):
    from cudagravitydemo_b200 import accuracy
    return accuracy.direct_sum(torch.from_numpy(p).cuda(), torch.from_numpy(t).cuda(), eps, 1.0).cpu().numpy()


def _potential(engine, torch, p, eps):
    v = torch.zeros((len(p), 3), device="cuda")
    return engine.diagnostics(torch.from_numpy(p).cuda(), v, eps, 1.0)["potential"]


def test_one_term_to_rounding(torch_cuda, engine):
    rng = np.random.default_rng(1)
    eps = 1e-40
    for e in np.concatenate([rng.uniform(-36, 37, 300), rng.uniform(-0.5, 0.5, 300)]):
        p = np.zeros((2, 4), np.float32)
        p[1, 0] = 10.0 ** e
        p[:, 3] = rng.uniform(0.5, 1, 2)
        d, m = np.longdouble(p[1, 0]), p[:, 3].astype(np.longdouble)
        r2 = d * d + np.longdouble(eps) ** 2
        want = m[1] * d / (r2 * np.sqrt(r2))
        got = _direct(torch_cuda, p, np.zeros(1, np.int32), eps)[0, 0]
        assert abs(got - want) <= TERM * want, e
        want = -m[0] * m[1] / np.sqrt(r2)
        assert abs(_potential(engine, torch_cuda, p, eps) - want) <= TERM * abs(want), e


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


@pytest.mark.parametrize("n", [26000, 40001, 51456, 65537])
def test_potential_over_several_tiles_a_block(torch_cuda, engine, n):
    """102, 157, 201 and 257 rows of bodies: from two row tiles a block up, with short last parts; the sums of
    some 1e3 positive terms a lane are good to 1e3 roundings."""
    torch = torch_cuda
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    p = torch.randn(n, 4, generator=g, device="cuda")
    p[:, 3] = torch.rand(n, generator=g, device="cuda") / n
    x, m = p[:, :3].double(), p[:, 3].double()
    want = 0.0
    for a in range(0, n, 2000):
        r2 = ((x[a:a + 2000, None, :] - x[None]) ** 2).sum(-1) + 0.01 ** 2
        w = m[a:a + 2000, None] * m[None] * torch.rsqrt(r2)
        k = torch.arange(w.shape[0], device="cuda")
        w[k, k + a] = 0.0
        want -= 0.5 * float(w.sum())
    got = engine.diagnostics(p, torch.zeros((n, 3), device="cuda"), 0.01, 1.0)["potential"]
    assert got == pytest.approx(want, rel=1e-12, abs=0)
