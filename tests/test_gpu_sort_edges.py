"""The radix sort at the edges of its tiles (4,096 pairs, 32 per warp and item),
of its one-cluster form (1,024 pairs per block, 16 blocks, one or two keys per
thread) and with digits that a warp shares wholly, partly or not at all."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 255, 256, 257, 1023, 1024, 1025, 4095, 4097, 16383, 16384, 16385, 18433, 32767, 32768, 32769,
         36864, 40961, 300007]


def _keys(rng, n, kind):
    if kind == "random":
        return rng.integers(0, 2 ** 64, n, dtype=np.uint64)
    if kind == "equal":
        return np.full(n, 0xFFFFFFFFFFFFFFFF, np.uint64)
    if kind == "two":
        return rng.choice(np.array([0xFF00FF00FF00FF00, 0x00FF00FF00FF00FF], np.uint64), n)
    if kind == "sorted":  # nearly, as a step's keys are
        return np.sort(rng.integers(0, 2 ** 63, n, dtype=np.uint64)) ^ rng.integers(0, 2 ** 20, n, dtype=np.uint64)
    return rng.integers(0, 300, n, dtype=np.uint64) << np.uint64(36)  # few values


@pytest.mark.parametrize("kind", ["random", "equal", "two", "sorted", "few"])
@pytest.mark.parametrize("n", SIZES)
def test_sort_edges(torch_cuda, engine, n, kind):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    k = _keys(rng, n, kind)
    v = rng.permutation(n).astype(np.uint32)
    lib = engine.lib()
    sorter = ctypes.c_void_p()
    assert lib.bh_sorter_create(ctypes.byref(sorter), n + 5) == 0
    kin = torch.from_numpy(k.view(np.int64)).cuda()
    vin = torch.from_numpy(v.view(np.int32)).cuda()
    kout, vout = torch.zeros_like(kin), torch.zeros_like(vin)
    try:
        for bits in (64, 45, 8):
            torch.cuda.synchronize()
            assert lib.bh_radix_sort_pairs(sorter, kin.data_ptr(), kout.data_ptr(), vin.data_ptr(), vout.data_ptr(), n,
                                           bits, None) == 0
            assert lib.bh_sorter_errors(sorter, None, None) == 0
            # whole 8-bit digits are sorted
            digits = k & np.uint64(2 ** (8 * ((bits + 7) // 8)) - 1)
            order = np.argsort(digits, kind="stable")
            assert np.array_equal(kout.cpu().numpy().view(np.uint64), k[order])
            assert np.array_equal(vout.cpu().numpy().view(np.uint32), v[order])
            assert np.array_equal(kin.cpu().numpy().view(np.uint64), k)
    finally:
        lib.bh_sorter_destroy(sorter)
