"""Results in pageable host memory around the size from which copies are
staged (8 MiB an array) and the ends of their 2 MiB chunks."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _roundtrip(n, seed):
    """A canonical block of n entries through get_ham_eff with an empty P."""
    from detnqs_b200 import core
    rng = np.random.default_rng(seed)
    row = np.repeat(np.arange(-(-n // 1024), dtype=np.uint32), 1024)[:n]
    col = (np.arange(n, dtype=np.uint32) % 1024) * 3
    val = rng.normal(size=n)
    got = core.get_ham_eff({"row": row, "col": col, "val": val, "shape": (4096, 4096)},
                           {"row": [], "col": [], "val": [], "shape": (0, 0)}, [], 0.0)
    np.testing.assert_array_equal(got["row"], row)
    np.testing.assert_array_equal(got["col"], col)
    np.testing.assert_array_equal(got["val"].view(np.uint64), val.view(np.uint64))


# values staged from 2^20 entries, rows and columns from 2^21
@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1, 1_310_721, 1 << 21,
                               (1 << 21) + 1, 4_000_003])
def test_sizes(n):
    _roundtrip(n, n)


def test_several_threads():
    errors = []

    def one(k):
        try:
            for q in range(3):
                _roundtrip(1_500_000 + 1000 * k + q, k)
        except Exception as e:   # reported by the main thread
            errors.append(e)

    team = [threading.Thread(target=one, args=(k,)) for k in range(4)]
    for t in team:
        t.start()
    for t in team:
        t.join()
    assert not errors, errors
