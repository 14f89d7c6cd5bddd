"""Radix sort at the edges of its three forms: one block, tiles of the grid
with one-word keys, and pairs packed into one word or taken word by word."""

import numpy as np
import pytest

from test_gpu_sort import _order

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 3583, 3584, 3585, 4095, 4096, 4097, 8193, 200_003])
@pytest.mark.parametrize("bits", [0, 1, 8, 9, 45, 64])
def test_one_word(n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << 63, size=n, dtype=np.uint64) * np.uint64(2) + \
        rng.integers(0, 2, size=n, dtype=np.uint64)
    keys = keys & np.uint64((1 << bits) - 1)
    keys[n // 2:] = keys[: n - n // 2]   # equal keys keep their order
    np.testing.assert_array_equal(_order(keys, [bits]), np.argsort(keys, kind="stable"))


# (20, 30): one packed word; (32, 32): its limit; (33, 32): word by word; a
# word without bits
@pytest.mark.parametrize("n", [1, 100, 3584, 3585, 50_001])
@pytest.mark.parametrize("bits", [(20, 30), (32, 32), (33, 32), (64, 64), (0, 17), (17, 0)])
def test_pairs(n, bits):
    rng = np.random.default_rng(n + bits[0])
    cols = [(rng.integers(0, 1 << 63, size=n, dtype=np.uint64) * np.uint64(2) +
             rng.integers(0, 2, size=n, dtype=np.uint64)) & np.uint64((1 << b) - 1) for b in bits]
    cols[0][n // 3:] = cols[0][: n - n // 3]
    np.testing.assert_array_equal(_order(np.stack(cols, 1), list(bits)),
                                  np.lexsort((cols[1], cols[0])))


# one tile, the few-tile scan and the three-phase scan of the row offsets:
# builds of these sizes return sorted blocks only if every offset is right
@pytest.mark.parametrize("dets", [2047, 2048, 8191, 8192, 8200])
def test_scan_sizes_through_a_build(dets):
    from detnqs_b200 import core, synthetic as S
    sysm = S.make_system(16, 6, 6, 32, 3)
    V = S.heat_bath_sample(sysm, dets, 3, max_level=4)
    assert len(V) == dets
    ctx = core.IntCtx.from_arrays(16, sysm.h1e, sysm.eri, sysm.e_core)
    got = core.get_ham_vv(V, ctx, 16)
    key = got["row"].astype(np.int64) * dets + got["col"]
    assert np.all(np.diff(key) > 0)
    assert np.array_equal(np.unique(got["row"]), np.arange(dets))
    # Hermitian with equal bits
    back = np.argsort(got["col"].astype(np.int64) * dets + got["row"], kind="stable")
    assert np.array_equal(got["val"][back].view(np.uint64), got["val"].view(np.uint64))
    ctx.close()
