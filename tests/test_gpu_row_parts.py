"""Candidate walks cut into parts of a row (few rows) or a row per warp (many)
against the oracle and the string-group build."""

import itertools

import numpy as np
import pytest

from conftest import assert_coo_equal
from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# one row (as many parts as pairs allow), a few, two electrons (one pair), and
# an odd count; rows of 40 orbitals keep both 64-bit halves busy
@pytest.mark.parametrize("n_orb,na,nb,dets", [(13, 5, 5, 1), (13, 5, 4, 37), (6, 1, 1, 20),
                                              (40, 7, 6, 5)])
def test_few_rows(port, n_orb, na, nb, dets):
    from detnqs_b200 import core
    sysm = S.make_system(n_orb, na, nb, 2 * n_orb, 9)
    V = np.ascontiguousarray(S.heat_bath_sample(sysm, dets, 4, max_level=3)) \
        if min(na, nb) > 1 else S.hf_sd_space(n_orb, na, nb)[:dets]
    psi = S.normalized_psi(len(V), 3)
    ctx = core.IntCtx.from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    chk = port.ctx_from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    chk.hb_prepare(1e-15)
    for got, want in ((core.get_ham_conn(V, ctx, n_orb, True, 1e-3),
                       chk.get_ham_conn(V, True, 1e-3)),
                      (core.get_ham_conn_amp(V, psi, ctx, n_orb, 1e-2),
                       chk.get_ham_conn_amp(V, psi, 1e-2))):
        assert_coo_equal(got["H_VV"], want["H_VV"])
        assert_coo_equal(got["H_VP"], want["H_VP"])
        np.testing.assert_array_equal(got["det_P"], want["det_P"])
    ctx.close()


def test_many_rows_take_a_row_per_warp():
    """15,876 determinants (all of 9 orbitals, 4a/4b): P is empty, H_VV is
    the string-group block bit for bit."""
    from detnqs_b200 import core
    sysm = S.make_system(9, 4, 4, 18, 2)
    strings = [sum(1 << o for o in c) for c in itertools.combinations(range(9), 4)]
    V = np.array([(a, b) for a in strings for b in strings], dtype=np.uint64)
    ctx = core.IntCtx.from_arrays(9, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    got = core.get_ham_conn(V, ctx, 9, True, 1e-15)
    assert got["size_P"] == 0 and len(got["H_VP"]["val"]) == 0
    assert_coo_equal(got["H_VV"], core.get_ham_vv(V, ctx, 9))
    ctx.close()


def test_local_connections_few_rows(port):
    from detnqs_b200 import core
    sysm = S.make_system(14, 6, 5, 28, 6)
    V = S.heat_bath_sample(sysm, 50, 6, max_level=3)
    ctx = core.IntCtx.from_arrays(14, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    chk = port.ctx_from_arrays(14, sysm.h1e, sysm.eri, sysm.e_core)
    chk.hb_prepare(1e-15)
    for hb in (True, False):
        got = core.get_local_connections(V, ctx, 14, hb, 1e-3)
        want = chk.get_local_connections(V, hb, 1e-3)
        np.testing.assert_array_equal(got["offsets"], want["offsets"])
        np.testing.assert_array_equal(got["dets"], want["dets"])
        np.testing.assert_array_equal(got["values"].view(np.uint64),
                                      want["values"].view(np.uint64))
    ctx.close()
