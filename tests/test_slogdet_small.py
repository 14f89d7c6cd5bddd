"""Log-det of small matrices at the edges of the row counts built, of the
matrices a warp holds, and with singular, tied and non-finite input."""

import numpy as np
import pytest

from test_slogdet import batch, reference

pytestmark = pytest.mark.gpu


# one matrix, a part-filled warp, and more than a block's worth; n up to and
# one past every built count
@pytest.mark.parametrize("n", [2, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 17, 20, 21, 24, 25, 32])
@pytest.mark.parametrize("B", [1, 3, 131])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_edges(n, B, dtype):
    from detnqs_b200 import slogdet as L
    rng = np.random.default_rng(100 * n + B)
    a = batch(rng, B, n, True, dtype)
    cot = rng.normal(size=B).astype(dtype)
    s0, l0, g0 = reference(a)
    s, l = L.slogdet(a)
    g = L.slogdet_grad(a, cot)
    eps = np.finfo(dtype).eps
    np.testing.assert_array_equal(s, s0)
    # backward error of LU: n eps per pivot on these well-conditioned matrices
    assert np.max(np.abs(l - l0)) <= 8 * n * n * eps
    want = cot[:, None, None] * g0
    assert np.max(np.abs(g - want)) <= 8 * n * n * eps * np.max(np.abs(want))


@pytest.mark.parametrize("n", [3, 10, 16])
def test_singular_tied_and_not_finite(n):
    """A zero column, equal rows, a NaN and an infinity beside sound matrices
    of the same warp; rows of equal magnitude (ties)."""
    from detnqs_b200 import slogdet as L
    rng = np.random.default_rng(n)
    a = batch(rng, 12, n)
    a[1, :, n - 1] = 0.0
    a[4, 2] = a[4, 0]
    a[6, 0, 0] = np.nan
    a[7, 1, 1] = np.inf
    a[9] = np.sign(rng.normal(size=(n, n)))   # ties in every column
    s, l = L.slogdet(a)
    g = L.slogdet_grad(a, np.ones(12))
    assert s[1] == 0 and l[1] == -np.inf and not np.any(g[1])
    ok = [0, 2, 3, 5, 8, 10, 11]
    s0, l0, g0 = reference(a[ok])
    np.testing.assert_array_equal(s[ok], s0)
    np.testing.assert_allclose(l[ok], l0, rtol=0, atol=1e-11)
    np.testing.assert_allclose(g[ok], g0, rtol=0, atol=1e-11 * np.max(np.abs(g0)))
    assert s[6] == 0 and l[6] == -np.inf and s[7] == 0 and l[7] == -np.inf
    s9, l9 = np.linalg.slogdet(a[9])
    if abs(s9) == 1 and l9 > -20:
        assert s[9] == s9 and abs(l[9] - l9) <= 1e-9
