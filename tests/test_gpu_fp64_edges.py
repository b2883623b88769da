"""The FP64 direct sum and the pair potential at the edges of their tiles (256
bodies), of their source splits and of their rows, against numpy.

Both sum at most n <= 5,000 terms of one sign or of mixed sign in double
precision; each term is within a few ulp and the sums within n ulp of their
magnitude sum, so 1e-11 of the magnitude sum bounds the difference with room."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _bodies(n, seed):
    rng = np.random.default_rng(seed)
    p = np.empty((n, 4), np.float32)
    p[:, :3] = rng.normal(0, 1, (n, 3)) * 10.0 ** rng.uniform(-3, 1, (n, 1))
    p[:, 3] = rng.uniform(0.1, 1, n) / n
    if n > 40:
        p[7, :3] = p[39, :3]  # a coincident pair
    return p


@pytest.mark.parametrize("nt", [1, 127, 256, 257, 1025])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1024, 1025, 2049, 5000])
def test_direct_sum_edges(torch_cuda, engine, n, nt):
    from cudagravitydemo_b200 import accuracy
    torch = torch_cuda
    p = _bodies(n, n)
    t = np.random.default_rng(nt).integers(0, n, nt).astype(np.int32)
    got = accuracy.direct_sum(torch.from_numpy(p).cuda(), torch.from_numpy(t).cuda(), 0.01, 2.0).cpu().numpy()
    x, m = p[:, :3].astype(np.float64), p[:, 3].astype(np.float64)
    for a in range(0, nt, 256):
        d = x[None] - x[t[a:a + 256]][:, None]
        f = 2.0 * m / ((d ** 2).sum(-1) + 0.01 ** 2) ** 1.5
        want, size = (f[..., None] * d).sum(1), (f[..., None] * np.abs(d)).sum(1)
        assert np.all(np.abs(got[a:a + 256] - want) <= TOL * size + 1e-300)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 511, 512, 513, 768, 1024, 1025, 1280, 3333, 5000])
def test_pair_potential_edges(torch_cuda, engine, n):
    torch = torch_cuda
    p = _bodies(n, n + 1)
    v = np.zeros((n, 3), np.float32)
    got = engine.diagnostics(torch.from_numpy(p).cuda(), torch.from_numpy(v).cuda(), 0.01, 2.0)["potential"]
    x, m = p[:, :3].astype(np.float64), p[:, 3].astype(np.float64)
    want = 0.0
    for i in range(0, n, 256):
        r = np.sqrt(((x[None] - x[i:i + 256][:, None]) ** 2).sum(-1) + 0.01 ** 2)
        w = m[None] * m[i:i + 256][:, None] / r
        w[np.arange(w.shape[0]), np.arange(i, i + w.shape[0])] = 0.0
        want -= w.sum()
    assert got == pytest.approx(want, rel=TOL, abs=0)


@pytest.mark.parametrize("n", [40, 300, 1000])
def test_infinite_and_zero_distances(torch_cuda, engine, n):
    from cudagravitydemo_b200 import accuracy
    torch = torch_cuda
    v = torch.zeros((n, 3), device="cuda")
    p = _bodies(n, n + 2)
    p[3, :3] = p[n - 1, :3]  # without softening a coincident pair is bound without limit
    assert engine.diagnostics(torch.from_numpy(p).cuda(), v, 0.0, 1.0)["potential"] == -np.inf
    far = _bodies(n, n + 2)
    far[n - 2, 0] = np.inf  # a body infinitely far away adds nothing
    gone = np.delete(far, n - 2, axis=0)
    got = engine.diagnostics(torch.from_numpy(far).cuda(), v, 0.01, 1.0)["potential"]
    want = engine.diagnostics(torch.from_numpy(gone).cuda(), v[1:], 0.01, 1.0)["potential"]
    assert got == pytest.approx(want, rel=TOL, abs=0)
    t = torch.arange(n, dtype=torch.int32, device="cuda")
    assert not accuracy.direct_sum(torch.from_numpy(p).cuda(), t, np.inf, 1.0).any()  # softened away
