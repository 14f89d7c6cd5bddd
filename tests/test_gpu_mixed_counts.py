"""Spaces that mix electron counts: strings that differ in two or four orbitals
without being excitations of each other connect nothing, whichever stage
evaluates the match."""

import numpy as np
import pytest

from conftest import assert_coo_equal
from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def _space(n, counts, each, seed):
    """Parts of the spaces of several (n_alpha, n_beta), shuffled."""
    rng = np.random.default_rng(seed)
    parts = []
    for na, nb in counts:
        V = S.hf_sd_space(n, na, nb)
        parts.append(V[rng.permutation(len(V))[:each]])
    V = np.concatenate(parts)
    return np.ascontiguousarray(V[rng.permutation(len(V))])


# counts 0, 1 and 2 apart in one spin and in both, an empty and a full string;
# strings of 32 bits and of 64
CASES = [(6, [(3, 3), (4, 3), (5, 3), (3, 1), (0, 0), (6, 6), (1, 5)], 60),
         (13, [(5, 5), (6, 5), (7, 5), (5, 3), (4, 4)], 150),
         (32, [(3, 2), (4, 2), (5, 2), (3, 4)], 150), (33, [(3, 2), (4, 2), (5, 2), (3, 4)], 150)]


@pytest.fixture(scope="module", params=CASES, ids=lambda c: f"{c[0]}o")
def system(port, request):
    from detnqs_b200 import core
    n, counts, each = request.param
    sysm = S.make_system(n, 2, 2, 2 * n, 9)
    V = _space(n, counts, each, n)
    ctx = core.IntCtx.from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    octx = port.ctx_from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    octx.hb_prepare(1e-15)
    yield ctx, octx, n, V, S.normalized_psi(len(V), 4)
    ctx.close()


def _want(octx, V, psi, policy):
    from detnqs_b200 import native as N
    if policy == N.POLICY_KNOWN_SETS:
        return octx.get_ham_vv(V)
    if policy == N.POLICY_STATIC:
        return octx.get_ham_conn(V, True, 1e-4)["H_VV"]
    return octx.get_ham_conn_amp(V, psi, 1e-4)["H_VV"]


# one pass, rows of more than a chunk, and the two-pass walk
@pytest.mark.parametrize("option,value", [(0, 0), ("OPT_ARENA_CHUNK", 8), ("OPT_ARENA_CAP", 64)])
@pytest.mark.parametrize("policy", ["POLICY_KNOWN_SETS", "POLICY_STATIC", "POLICY_DYNAMIC"])
def test_builds(system, policy, option, value):
    from detnqs_b200 import device, native as N
    ctx, octx, n, V, psi = system
    pol = getattr(N, policy)
    if option:
        N.check(N.lib.dnq_set_option(getattr(N, option), value))
    try:
        H = device.build(ctx, V, n_orb=n, policy=pol, use_heatbath=True, eps1=1e-4, psi=psi,
                         want_vp=False)
        got = H.to_coo(0)
        H.close()
    finally:
        if option:
            N.check(N.lib.dnq_set_option(getattr(N, option), 0))
    assert_coo_equal(got, _want(octx, V, psi, pol))


def test_batch_and_energy(system):
    from detnqs_b200 import core, native as N
    from detnqs_b200.batch import Batch
    ctx, octx, n, V, psi = system
    pure = np.ascontiguousarray(S.hf_sd_space(n, 2, 2)[:100])
    b = Batch([ctx, ctx], [V, pure], [n, n], policy=N.POLICY_STATIC, use_heatbath=True, eps1=1e-4)
    b.step(np.concatenate([psi, np.ones(len(pure))]), precision=N.F64)
    assert_coo_equal(b.coo(0), octx.get_ham_conn(V, True, 1e-4)["H_VV"])
    assert_coo_equal(b.coo(1), octx.get_ham_conn(pure, True, 1e-4)["H_VV"])
    b.close()
    e = core.compute_variational_energy(V, psi, ctx, n, True, 1e-4)
    e0 = octx.compute_variational_energy(V, psi, True, 1e-4)
    assert abs(e - e0) <= 1e-12 * max(1.0, abs(e0))
