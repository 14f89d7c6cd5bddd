"""Spaces of fewer orbitals than the integral context holds: no ket may take
an orbital past n_orb (ham_utils.cpp:470-479), whatever the pair table of the
context lists, so blocks, generators, connections, energy and PT2 equal the
oracle's."""

import numpy as np
import pytest

from conftest import assert_coo_equal
from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# strings packed into one word by n_orb and by the context; one word for the
# space only (32 of 33); two words
@pytest.fixture(scope="module", params=[(13, 10, 4, 3), (13, 12, 5, 5), (33, 32, 3, 2),
                                        (36, 33, 2, 3)], ids=lambda p: f"{p[1]}of{p[0]}")
def space(port, request):
    from detnqs_b200 import core
    n, n_orb, na, nb = request.param
    sysm = S.make_system(n, na, nb, 2 * n, 11)
    V = S.hf_sd_space(n_orb, na, nb)
    V = np.ascontiguousarray(V[np.linspace(0, len(V) - 1, 24).astype(int)])
    ctx = core.IntCtx.from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    octx = port.ctx_from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    octx.hb_prepare(1e-15)
    octx.n_orb = n_orb
    yield core, ctx, octx, V, S.normalized_psi(len(V), 5), n_orb
    ctx.close()


def _same_blocks(got, want):
    assert_coo_equal(got["H_VV"], want["H_VV"])
    assert_coo_equal(got["H_VP"], want["H_VP"])
    np.testing.assert_array_equal(got["det_P"], want["det_P"])


@pytest.mark.parametrize("use_hb", [True, False])
def test_connected_blocks(space, use_hb):
    core, ctx, octx, V, psi, n_orb = space
    _same_blocks(core.get_ham_conn(V, ctx, n_orb, use_hb, 1e-4),
                 octx.get_ham_conn(V, use_hb, 1e-4))


def test_amplitude_blocks(space):
    core, ctx, octx, V, psi, n_orb = space
    _same_blocks(core.get_ham_conn_amp(V, psi, ctx, n_orb, 1e-4),
                 octx.get_ham_conn_amp(V, psi, 1e-4))


@pytest.mark.parametrize("mode", ["none", "static", "dynamic"])
def test_generators(space, mode):
    core, ctx, octx, V, psi, n_orb = space
    np.testing.assert_array_equal(
        core.gen_perturbative_dets(V, n_orb, ctx, psi, mode=mode, eps1=1e-4),
        octx.gen_perturbative_dets(V, psi, mode, 1e-4))


@pytest.mark.parametrize("use_hb", [True, False])
def test_local_connections(space, use_hb):
    core, ctx, octx, V, psi, n_orb = space
    got = core.get_local_connections(V, ctx, n_orb, use_hb, 1e-4)
    want = octx.get_local_connections(V, use_hb, 1e-4)
    for key in ("offsets", "dets", "values"):
        np.testing.assert_array_equal(got[key], want[key])


@pytest.mark.parametrize("use_hb", [True, False])
def test_energy_and_pt2(space, use_hb):
    core, ctx, octx, V, psi, n_orb = space
    e = core.compute_variational_energy(V, psi, ctx, n_orb, use_hb, 1e-4)
    e0 = octx.compute_variational_energy(V, psi, use_hb, 1e-4)
    assert abs(e - e0) <= 1e-12 * max(1.0, abs(e0))
    got = core.compute_pt2(V, psi, ctx, n_orb, -50.0, use_hb, 1e-5)
    want = octx.compute_pt2(V, psi, -50.0, use_hb, 1e-5)
    assert got["n_ext"] == want["n_ext"]
    for part in ("e_pt2_external", "e_pt2_internal"):
        assert abs(got[part] - want[part]) <= 1e-12 * max(1.0, abs(want[part]))


# large enough for the string groups (builds of V alone, energy, batch), in
# one word and in two
@pytest.mark.parametrize("n,n_orb", [(20, 16), (36, 33)])
def test_string_groups(port, n, n_orb):
    from detnqs_b200 import core, native as N
    from detnqs_b200.batch import Batch
    sysm = S.make_system(n, 4, 4, 2 * n, 3)
    V = np.ascontiguousarray(S.hf_sd_space(n_orb, 4, 4)[:2500])
    psi = S.normalized_psi(len(V), 1)
    ctx = core.IntCtx.from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)
    octx = port.ctx_from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    octx.hb_prepare(1e-15)
    octx.n_orb = n_orb
    want = octx.get_ham_vv(V)
    assert_coo_equal(core.get_ham_vv(V, ctx, n_orb), want)
    b = Batch([ctx], [V], [n_orb], policy=N.POLICY_KNOWN_SETS, use_heatbath=False, eps1=0.0)
    assert_coo_equal(b.coo(0), want)
    b.close()
    e = core.compute_variational_energy(V, psi, ctx, n_orb, True, 1e-5)
    e0 = octx.compute_variational_energy(V, psi, True, 1e-5)
    assert abs(e - e0) <= 1e-12 * max(1.0, abs(e0))
    ctx.close()
