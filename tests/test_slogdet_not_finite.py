"""A matrix with NaN leaves the other matrices of its warp, of the next warp
and of the block's last warp alone, and its own value and gradient are those
of a singular one."""

import numpy as np
import pytest

from test_slogdet import batch, reference

pytestmark = pytest.mark.gpu


# a warp holds 8 matrices up to n = 4, 4 up to 8, 2 up to 16 and one above;
# a block four times as many.  NaN in every position of a warp, sound
# matrices before and after it
@pytest.mark.parametrize("n", [2, 4, 5, 8, 10, 16, 17, 24, 32])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("where", ["first", "last", "column"])
def test_neighbours_of_nan(n, dtype, where):
    from detnqs_b200 import slogdet as L
    rng = np.random.default_rng(n)
    B = 67
    a = batch(rng, B, n, True, dtype)
    bad = np.arange(0, B, 3)   # every place of 2, 4 and 8 a warp in turn
    if where == "first":
        a[bad, 0, 0] = np.nan
    elif where == "last":
        a[bad, n - 1, n - 1] = np.nan
    else:
        a[bad, :, n // 2] = np.nan
    cot = rng.normal(size=B).astype(dtype)
    s, l = L.slogdet(a)
    g = L.slogdet_grad(a, cot)
    assert not np.any(s[bad]) and np.all(l[bad] == -np.inf) and not np.any(g[bad])
    ok = np.setdiff1d(np.arange(B), bad)
    s0, l0, g0 = reference(a[ok])
    eps = np.finfo(dtype).eps
    np.testing.assert_array_equal(s[ok], s0)
    # backward error of LU: n eps per pivot on these well-conditioned matrices
    assert np.max(np.abs(l[ok] - l0)) <= 8 * n * n * eps
    want = cot[ok][:, None, None] * g0
    assert np.max(np.abs(g[ok] - want)) <= 8 * n * n * eps * np.max(np.abs(want))
    # and bit for bit what the sound matrices give by themselves
    np.testing.assert_array_equal(g[ok], L.slogdet_grad(np.ascontiguousarray(a[ok]), cot[ok]))
