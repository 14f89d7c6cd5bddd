"""External PT2 sums over sorted contributions: keys of one word (up to 32
orbitals) and of two, runs within and across tiles, against the oracle."""

import numpy as np
import pytest

from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# one row (every run has one entry), fewer contributions than a tile, many
# (runs cross tiles); 32 orbitals fill a key word, 33 take two
@pytest.mark.parametrize("n_orb,na,nb,dets", [(6, 2, 1, 3), (13, 5, 4, 1), (13, 5, 5, 300),
                                              (32, 3, 2, 20), (33, 3, 2, 20)])
@pytest.mark.parametrize("use_hb", [False, True])
def test_external_sum(port, n_orb, na, nb, dets, use_hb):
    from detnqs_b200 import core
    sysm = S.make_system(n_orb, na, nb, 2 * n_orb, 9)
    V = S.hf_sd_space(n_orb, na, nb)
    V = np.ascontiguousarray(V[np.linspace(0, len(V) - 1, dets).astype(int)])
    psi = S.normalized_psi(len(V), 3)
    e_ref = -50.0
    ctx = core.IntCtx.from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    chk = port.ctx_from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    chk.hb_prepare(1e-15)
    got = core.compute_pt2(V, psi, ctx, n_orb, e_ref, use_hb, 1e-6)
    want = chk.compute_pt2(V, psi, e_ref, use_hb, 1e-6)
    assert got["n_ext"] == want["n_ext"]
    for part in ("e_pt2_external", "e_pt2_internal"):
        assert abs(got[part] - want[part]) <= 1e-12 * max(1.0, abs(want[part]))
    ctx.close()


@pytest.mark.parametrize("n_orb", [31, 32, 33])
def test_diagonal_elements(port, n_orb):
    """Strings of 32 bits and of 64: bit for bit."""
    from detnqs_b200 import core
    sysm = S.make_system(n_orb, 5, 4, 2 * n_orb, 4)
    rng = np.random.default_rng(n_orb)
    V = np.array([[sum(1 << int(o) for o in rng.choice(n_orb, k, replace=False))
                   for k in rng.integers(0, n_orb + 1, 2)] for _ in range(200)], dtype=np.uint64)
    ctx = core.IntCtx.from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    chk = port.ctx_from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    np.testing.assert_array_equal(core.get_ham_diag(V, ctx), chk.get_ham_diag(V))
    ctx.close()
