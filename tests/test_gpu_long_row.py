"""Diagonal element of an H_VP row with very many entries: the FP64 sum has
the rounding of one addition after the other."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _terms(kind, n):
    """(a, d): amplitudes and denominators; a term is (a * (1 / d)) * a."""
    rng = np.random.default_rng(n)
    a = rng.normal(size=n)
    d = -1.0 - 9.0 * rng.random(n)
    if kind == "alternating":      # the sum turns and passes zero
        d *= rng.choice((-1.0, 1.0), n)
    elif kind == "ties":           # every rounding is half way now and then
        a = 2.0 ** rng.integers(-30, 1, n)
        d = -(2.0 ** rng.integers(-20, 21, n))
    elif kind == "growing":        # a new binade every few terms, then small ones
        a = np.concatenate([2.0 ** (np.arange(400) / 3.0 - 60.0), a[400:] * 1e-3])
    elif kind == "zeros":          # a screened-out stretch first
        a[: n // 2] = 1e-9
    elif kind == "cancelling":     # pairs that cancel exactly
        a[1::2] = a[: n - n % 2: 2]
        d[1::2] = -d[: n - n % 2: 2]
    elif kind == "nan":
        a[n // 3] = np.nan
    return a, d


# one entry past the long-row limit, and ragged last tiles
@pytest.mark.parametrize("n", [65_537, 69_632, 200_001])
@pytest.mark.parametrize("kind", ["same_sign", "alternating", "ties", "growing", "zeros",
                                  "cancelling", "nan"])
def test_sum_keeps_the_order_of_additions(kind, n):
    from detnqs_b200 import core
    a, d = _terms(kind, n)
    vv = {"row": np.zeros(1, np.uint32), "col": np.zeros(1, np.uint32), "val": np.zeros(1) + 0.5,
          "shape": (1, 1)}
    vp = {"row": np.zeros(n, np.uint32), "col": np.arange(n, dtype=np.uint32), "val": a,
          "shape": (1, n)}
    got = core.get_ham_eff(vv, vp, -d, 0.0, reg_type="linear_shift", epsilon=0.0)
    dinv = 1.0 / d
    keep = ~(np.abs(dinv) * (a * a) < 1e-12) & ~(a == 0.0)
    want = np.cumsum(np.concatenate([[0.0], ((a * dinv) * a)[keep]]))[-1] + 0.5
    if np.isnan(want):
        assert len(got["val"]) == 0 or np.isnan(got["val"][0])
    else:
        assert got["val"].view(np.uint64)[0] == np.array([want]).view(np.uint64)[0]
