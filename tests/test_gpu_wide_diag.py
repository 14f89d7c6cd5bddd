"""Diagonal elements of two-word determinants: many at once (tables staged in
shared memory) and few, bit for bit, against the oracle."""

import numpy as np
import pytest

from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# one word, strings that end in the second, third and fourth 32 bits; more
# elements than threads, with a ragged last round
@pytest.mark.parametrize("n_orb", [7, 33, 64, 70, 97])
def test_many_equal_few(n_orb):
    from detnqs_b200 import wide as Wd
    from oracle import WideChecker
    sysm = S.make_system(n_orb, 3, 2, 8, 5)
    rng = np.random.default_rng(n_orb)
    n = 200_003
    d = np.zeros((n, 4), np.uint64)
    for k in range(2):
        # any electron count, empty and full strings included
        p = rng.random((n, 1)) * 1.2 - 0.1
        occ = rng.random((n, n_orb)) < p
        for o in range(n_orb):
            d[:, 2 * k + o // 64] |= occ[:, o].astype(np.uint64) << np.uint64(o % 64)
    ctx = Wd.IntCtxWide.from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    got = Wd.get_ham_diag_wide(d, ctx)
    few = np.concatenate([Wd.get_ham_diag_wide(np.ascontiguousarray(x), ctx)
                          for x in np.array_split(d, 20)])
    assert np.array_equal(got.view(np.uint64), few.view(np.uint64))
    chk = WideChecker(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    x = np.ascontiguousarray(d[::1000])
    assert np.array_equal(got[::1000].view(np.uint64), chk.diag(x).view(np.uint64))
    ctx.close()
