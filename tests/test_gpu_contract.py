"""Matrix-free contraction (variational energy, internal PT2 part) by string
groups against the candidate walk and the oracle."""

import numpy as np
import pytest

from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def _system(n_orb, ne, dets, seed=5):
    sysm = S.make_system(n_orb, ne, ne, 2 * n_orb, seed)
    V = S.heat_bath_sample(sysm, dets, seed, max_level=3)
    rng = np.random.default_rng(seed)
    psi = rng.normal(size=len(V)) * 10.0 ** (-2.0 * rng.random(len(V)))
    return sysm, V, psi / np.linalg.norm(psi)


def _both(core, N, V, psi, ctx, n_orb, use_hb, eps):
    """(string groups where the rule picks them, candidate walk)."""
    got = core.compute_variational_energy(V, psi, ctx, n_orb, use_hb, eps)
    N.check(N.lib.dnq_set_option(N.OPT_FORCE_WALK, 1))
    try:
        walk = core.compute_variational_energy(V, psi, ctx, n_orb, use_hb, eps)
    finally:
        N.check(N.lib.dnq_set_option(N.OPT_FORCE_WALK, 0))
    return got, walk


# 1 and 2 rows, one short of and past a block of rows, u32 and u64 strings,
# rows cut into slices (the reference row of 3001) and spaces with a spin of
# one electron
@pytest.mark.parametrize("n_orb,ne,dets", [(30, 12, 1), (30, 12, 2), (30, 12, 257), (32, 13, 900),
                                           (33, 13, 900), (28, 11, 3001), (60, 1, 1500)])
@pytest.mark.parametrize("use_hb,eps", [(True, 1e-3), (False, 1e-6)])
def test_energy_matches_walk_and_oracle(port, n_orb, ne, dets, use_hb, eps):
    from detnqs_b200 import core, native as N
    sysm, V, psi = _system(n_orb, ne, dets)
    ctx = core.IntCtx.from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    got, walk = _both(core, N, V, psi, ctx, n_orb, use_hb, eps)
    # both sum with Dot2: the rounded results are neighbours at most
    assert abs(got - walk) <= 4 * np.spacing(abs(walk))
    if dets <= 900:
        octx = port.ctx_from_arrays(n_orb, sysm.h1e, sysm.eri, sysm.e_core)
        octx.hb_prepare(1e-15)
        want = octx.compute_variational_energy(V, psi, use_hb, eps)
        assert abs(got - want) <= 1e-12 * max(1.0, abs(want))
    ctx.close()


def test_duplicates_and_mixed_electron_counts_keep_their_meaning():
    """A repeated determinant and a basis of several electron counts take the
    walk's rules (amplitudes by de-duplicated position; only equal counts
    connect)."""
    from detnqs_b200 import core, native as N
    sysm, V, psi = _system(28, 11, 400)
    ctx = core.IntCtx.from_arrays(28, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    dup = np.concatenate([V, V[5:9]])
    rng = np.random.default_rng(1)
    for basis in (dup, np.concatenate([V, V[:60] | np.uint64(1 << 27), S.hf_determinant(9, 13)])):
        basis = np.ascontiguousarray(basis)
        c = rng.normal(size=len(basis))
        got, walk = _both(core, N, basis, c, ctx, 28, True, 1e-4)
        assert abs(got - walk) <= 4 * np.spacing(abs(walk))
    ctx.close()


def test_pt2_internal_part_matches_walk():
    from detnqs_b200 import core, native as N
    sysm, V, psi = _system(28, 11, 900)
    ctx = core.IntCtx.from_arrays(28, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    e_ref = float(core.get_ham_diag(V[:1], ctx)[0]) - 0.5
    got = core.compute_pt2(V, psi, ctx, 28, e_ref, True, 1e-2)
    N.check(N.lib.dnq_set_option(N.OPT_FORCE_WALK, 1))
    try:
        walk = core.compute_pt2(V, psi, ctx, 28, e_ref, True, 1e-2)
    finally:
        N.check(N.lib.dnq_set_option(N.OPT_FORCE_WALK, 0))
    # r_i = sigma_i - e_ref c_i, both from neighbouring sigma
    assert abs(got["e_pt2_internal"] - walk["e_pt2_internal"]) <= 1e-12 * abs(
        walk["e_pt2_internal"])
    assert got["n_ext"] == walk["n_ext"]
    ctx.close()
