"""The page-locked slots of the staged copies: made only under a context that
keeps them, shared by threads, and given back with the last context."""

import os
import subprocess
import sys
import threading

import pytest

from test_gpu_host_copies import _roundtrip

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# copies of n entries into arrays in use, without a context: just below the
# size that is staged, and twice that
_NO_CONTEXT = """
import ctypes as C
import time
import numpy as np
from detnqs_b200 import native as N

def run(n):
    row = np.repeat(np.arange(n // 1024, dtype=np.uint32), 1024)
    col = (np.arange(n, dtype=np.uint32) % 1024) * 3
    val = np.ones(n)
    h = C.c_void_p()
    N.check(N.lib.dnq_ham_eff(row.ctypes.data, col.ctypes.data, val.ctypes.data, n, 4096, None,
                              None, None, 0, 0, None, 0.0, 1, 1e-12, N.F64, 0, None, C.byref(h)))
    t = []
    for k in range(16):
        t0 = time.perf_counter()
        N.check(N.lib.dnq_ham_copy_coo(h, 0, row.ctypes.data, col.ctypes.data, val.ctypes.data,
                                       None))
        t.append(time.perf_counter() - t0)
    N.check(N.lib.dnq_ham_destroy(h))
    return sorted(t[1:])[7]

run(1 << 20)
print(run((1 << 20) - 1024), run(1 << 21))
"""


def test_no_context_makes_no_slots():
    """Twice the bytes take about twice the time; locking and releasing the
    slots for every copy made it tens of times."""
    r = subprocess.run([sys.executable, "-c", _NO_CONTEXT], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    below, above = map(float, r.stdout.split())
    assert above <= 8 * below, (below, above)


def _context():
    from detnqs_b200 import core
    from detnqs_b200 import synthetic as S
    sysm = S.make_system(6, 2, 2, 12, 1)
    return core.IntCtx.from_arrays(6, sysm.h1e, sysm.eri, sysm.e_core)


# the sizes of the unstaged copies again, after enough bytes that the slots
# are made; and from more threads than there are slot sets
def test_sizes_under_a_context():
    ctx = _context()
    for k in range(5):
        _roundtrip(4_000_003 + k, k)   # 64 MB each
    for n in ((1 << 20) - 1, 1 << 20, (1 << 20) + 1, 1_310_721, 1 << 21, (1 << 21) + 1):
        _roundtrip(n, n)
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
    ctx.close()
    _roundtrip(1 << 21, 7)
    ctx = _context()
    _roundtrip(1 << 21, 8)
    ctx.close()
