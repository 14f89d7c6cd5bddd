"""What the framework does for its users, as cases that can be timed.

A selected-CI program with a neural ansatz calls this framework for
screened H_VV builds and local energies, H.psi on resident blocks, proxy
blocks (V plus discovered P) and their downfolding, matrix-free energies and
PT2, batches of systems, batch features of determinants and the log-det of
its orbital matrices.  Every case is one such call through the public Python
entry points, on seeded synthetic integrals (symmetric h, Cholesky-form
positive semi-definite ERIs) and heat-bath sampled determinant spaces.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and the handles a program keeps
    run(state)          one pass
    work(case)          bytes and flops a pass cannot do without
    exact(case, seed)   the outputs in 64 bits, from plain torch
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from detnqs_b200 import core, det_utils, device, native, operator, slogdet, wide
from detnqs_b200.batch import Batch

DEV = "cuda"
F64 = torch.float64
I64 = torch.int64


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # The smallest build of a selected-CI loop: HF plus all singles and
        # doubles of 5a/5b electrons in 13 orbitals, every double kept, and
        # the local energies on it.  Launches and latency count.
        dict(name="vv_full_13o_2241", kind="vv_full", n_orb=13, n_el=5, dets=2241, space="sd"),
        # The largest build: 30 orbitals, 12a/12b, 1e6 determinants, static
        # heat-bath screening, then FP64 and FP32 local energies.
        dict(name="vv_static_30o_1e6", kind="vv_static", n_orb=30, n_el=12, dets=1_000_000,
             level=4, eps1=1e-6),
        # H on 8 amplitude vectors at once, on a resident block of an odd size.
        dict(name="hpsi_f32_k8_30o_200003", kind="hpsi", n_orb=30, n_el=12, dets=200_003, level=4,
             k=8, fp32=True),
        # One outer iteration with discovered P: proxy build, diag(H_PP),
        # downfolding and H_eff.psi for the 13-orbital space.
        dict(name="proxy_eff_13o_2241", kind="proxy_eff", n_orb=13, n_el=5, dets=2241, space="sd",
             screening="static", eps1=1e-6, fp32=False),
        # The inner loop on a resident proxy: H_VV, H_VP and H_PV products.
        dict(name="proxy_apply_20o_3001", kind="proxy_apply", n_orb=20, n_el=8, dets=3001, level=4,
             eps1=1e-4, fp32=False),
        # The drop-in builder with amplitude screening, blocks returned to
        # the host in the reference's COO format.
        dict(name="conn_amp_24o_403", kind="conn_amp", n_orb=24, n_el=9, dets=403, level=4,
             eps1=1e-4),
        # Variational energy of a fixed basis without keeping a matrix.
        dict(name="energy_30o_20011", kind="energy", n_orb=30, n_el=12, dets=20_011, level=4,
             heatbath=True, eps1=1e-6),
        # Perturbative correction of a converged space.
        dict(name="pt2_20o_3001", kind="pt2", n_orb=20, n_el=8, dets=3001, level=4, heatbath=True,
             eps1=1e-4),
        # Downfolding beyond 64 orbitals (two words per spin string).
        dict(name="wide_eff_100o_10007", kind="wide_eff", n_orb=100, n_el=20, dets=10_007, level=4,
             eps1=1e-5, fp32=False),
        # Many systems of uneven size rebuilt and contracted in one step.
        dict(name="batch_step_12", kind="batch", systems=12, dets=30_000, fp32=True),
        # Network inputs of a whole space: occupations, ranks, signs, holes,
        # particles and their positions.
        dict(name="features_30o_1e6", kind="features", n_orb=30, n_el=12, dets=1_000_003, kmax=8,
             phase=True, positions=True),
        # The ansatz' determinants, forward and backward.
        dict(name="slogdet_10x10_32768", kind="slogdet", n=10, batch=32_768, fp32=False),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _electrons(rng, n_orb):
    """An electron count per spin between 40% and 60% filling."""
    return rng.randint(math.ceil(0.4 * n_orb), math.floor(0.6 * n_orb))


KINDS = ("vv_full", "vv_static", "hpsi", "proxy_eff", "proxy_apply", "conn_amp", "energy", "pt2",
         "wide_eff", "batch", "features", "slogdet")


def draw(rng):
    kind = rng.choice(KINDS)
    c = dict(kind=kind)
    if kind in ("vv_full", "vv_static", "hpsi", "energy"):
        n = rng.randint(14, 32)
        c.update(n_orb=n, n_el=_electrons(rng, n), level=rng.choice((3, 4)))
    if kind == "vv_full":
        c.update(dets=_log_uniform(rng, 500, 20_000))
    elif kind == "vv_static":
        c.update(dets=_log_uniform(rng, 1_000, 300_000), eps1=10.0 ** rng.randint(-7, -3))
    elif kind == "hpsi":
        c.update(dets=_log_uniform(rng, 5_000, 200_003), k=rng.randint(1, 12),
                 fp32=rng.random() < 0.5)
    elif kind == "energy":
        c.update(dets=_log_uniform(rng, 500, 20_000), heatbath=rng.random() < 0.7,
                 eps1=10.0 ** rng.randint(-6, -3))
    elif kind in ("proxy_eff", "proxy_apply"):
        n = rng.randint(10, 20)
        c.update(n_orb=n, n_el=max(2, int(0.4 * n)), dets=_log_uniform(rng, 200, 2_000), level=4,
                 eps1=10.0 ** rng.randint(-6, -3), fp32=rng.random() < 0.5)
        if kind == "proxy_eff":
            c.update(screening=rng.choice(("static", "dynamic")))
    elif kind == "conn_amp":
        n = rng.randint(12, 24)
        c.update(n_orb=n, n_el=max(2, int(0.4 * n)), dets=_log_uniform(rng, 50, 400), level=4,
                 eps1=10.0 ** rng.randint(-5, -3))
    elif kind == "pt2":
        n = rng.randint(12, 20)
        c.update(n_orb=n, n_el=max(2, int(0.4 * n)), dets=_log_uniform(rng, 200, 3_000), level=4,
                 heatbath=rng.random() < 0.7, eps1=10.0 ** rng.randint(-5, -3))
    elif kind == "wide_eff":
        c.update(n_orb=rng.randint(66, 100), n_el=rng.randint(10, 20),
                 dets=_log_uniform(rng, 1_000, 10_000), level=4, eps1=1e-5,
                 fp32=rng.random() < 0.5)
    elif kind == "batch":
        c.update(systems=rng.randint(3, 12), dets=_log_uniform(rng, 3_000, 30_000),
                 fp32=rng.random() < 0.5)
    elif kind == "features":
        n = rng.randint(8, 60)
        c.update(n_orb=n, n_el=_electrons(rng, n), dets=_log_uniform(rng, 1_000, 1_000_000),
                 kmax=rng.choice((0, 4, 5, 8)), phase=rng.random() < 0.5,
                 positions=rng.random() < 0.5)
    elif kind == "slogdet":
        n = rng.randint(2, 64)
        c.update(n=n, batch=_log_uniform(rng, 256, max(1_024, 3_000_000 // (n * n))),
                 fp32=rng.random() < 0.5)
    return c


# ---------------------------------------------------------------------------
# Inputs: integrals, determinant spaces, amplitudes
# ---------------------------------------------------------------------------

def _integrals(n, seed):
    """Packed (h1e, eri): diag(h) ~ U(-20, 0) ascending, off-diagonals
    N(0, 0.05), (pq|rs) = sum_K L_pq L_rs with 2n vectors of N(0, 0.1)."""
    rng = np.random.default_rng(seed)
    n1 = n * (n + 1) // 2
    h = rng.normal(0.0, 0.05, n1)
    h[np.cumsum(np.arange(1, n + 1)) - 1] = np.sort(rng.uniform(-20.0, 0.0, n))
    L = torch.from_numpy(rng.normal(0.0, 0.1, (2 * n, n1))).to(DEV)
    G = L.T @ L
    i, j = torch.tril_indices(n1, n1, device=DEV)
    return h, G[i, j].cpu().numpy()


def _dense(h, eri, n):
    """Full h[p, q] and (pq|rs) on the GPU."""
    p = torch.arange(n, device=DEV)
    hi, lo = torch.maximum(p[:, None], p[None]), torch.minimum(p[:, None], p[None])
    key = hi * (hi + 1) // 2 + lo
    k1, k2 = key[:, :, None, None], key[None, None]
    hi, lo = torch.maximum(k1, k2), torch.minimum(k1, k2)
    flat = torch.from_numpy(eri).to(DEV)[hi * (hi + 1) // 2 + lo]
    return torch.from_numpy(h).to(DEV)[key], flat


def _words(occ):
    """bool[N, n] -> int64[N, ceil(n / 64)] bit masks, low word first."""
    out = []
    for lo in range(0, occ.shape[1], 64):
        part = occ[:, lo:lo + 64]
        sh = torch.arange(part.shape[1], device=occ.device)
        out.append((part.to(I64) << sh).sum(1))
    return torch.stack(out, 1)


def _keys(a, b):
    """One 64-bit key per determinant (its words through odd multipliers)."""
    w = torch.cat([_words(a), _words(b)], 1)
    mul = torch.tensor([-7046029254386353131, 1609587929392839161, -4417276706812531889,
                        2870177450012600261], device=DEV)
    return (w * mul[:w.shape[1]]).sum(1)


def _masks(a, b, two_words=False):
    """uint64[N, 2] (or [N, 4]) determinants on the host."""
    wa, wb = _words(a), _words(b)
    if two_words and wa.shape[1] == 1:
        wa, wb = (torch.cat([w, torch.zeros_like(w)], 1) for w in (wa, wb))
    return torch.cat([wa, wb], 1).cpu().numpy().view(np.uint64)


def _level(a, b, na, nb):
    return (~a[:, :na]).sum(1) + (~b[:, :nb]).sum(1)


def _sample(eri4, n, na, nb, count, level, seed):
    """Heat-bath sampling from HF: uniform parents of the set so far, 1 in
    16 proposals a uniform single, else a double of a uniform occupied pair
    (same spin 5 in 15) with its virtual pair drawn by |<ij||ab>|; children
    up to `level` excitations, kept in draw order.  bool[N, n] per spin."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    nn = n * n

    def cdf(w):
        cs = torch.cumsum(w.reshape(nn, nn), 1)
        tot = cs[:, -1].clone()
        base = torch.cumsum(tot, 0) - tot
        return (cs + base[:, None]).reshape(-1), base, tot

    x = eri4.permute(0, 2, 1, 3)
    os_ = cdf(x.abs())
    ss = cdf((x - eri4.permute(0, 2, 3, 1)).abs() * torch.ones(n, n, device=DEV).triu(1))
    a = torch.zeros(1, n, dtype=torch.bool, device=DEV)
    b = a.clone()
    a[:, :na] = True
    b[:, :nb] = True
    m = 1 << 18

    def rand(k):
        return torch.randint(0, k, (m,), generator=g, device=DEV)

    def pick(table, row):
        flat, base, tot = table
        u = base[row] + torch.rand(m, generator=g, device=DEV, dtype=F64) * tot[row]
        k = (torch.searchsorted(flat, u, right=True) - row * nn).clamp(0, nn - 1)
        return k // n, k % n

    r = torch.arange(m, device=DEV)
    while True:
        before = len(a)
        par = rand(before)
        pa, pb = a[par].clone(), b[par].clone()
        oa = pa.nonzero()[:, 1].view(m, na)
        ob = pb.nonzero()[:, 1].view(m, nb)
        kind, spin = rand(16), rand(2) == 0
        i, j = oa[r, rand(na)], ob[r, rand(nb)]
        ta, tb = pick(os_, i * n + j)
        os_ok = (kind > 5) & ~pa[r, ta] & ~pb[r, tb]
        ps = torch.where(spin[:, None], pa, pb)
        o = torch.where(spin[:, None], oa, ob)
        q = rand(na)
        s1, s2 = o[r, q], o[r, (q + 1 + rand(max(na - 1, 1))) % na]
        t1, t2 = pick(ss, torch.minimum(s1, s2) * n + torch.maximum(s1, s2))
        ss_ok = (kind > 0) & (kind <= 5) & (s1 != s2) & (t1 != t2) & ~ps[r, t1] & ~ps[r, t2]
        h, p = o[r, rand(na)], rand(n)
        s_ok = (kind == 0) & ~ps[r, p]
        pa[r[os_ok], i[os_ok]] = False
        pa[r[os_ok], ta[os_ok]] = True
        pb[r[os_ok], j[os_ok]] = False
        pb[r[os_ok], tb[os_ok]] = True
        for X, sp in ((pa, spin), (pb, ~spin)):
            d, s = ss_ok & sp, s_ok & sp
            X[r[d], s1[d]] = False
            X[r[d], s2[d]] = False
            X[r[d], t1[d]] = True
            X[r[d], t2[d]] = True
            X[r[s], h[s]] = False
            X[r[s], p[s]] = True
        ok = (os_ok | ss_ok | s_ok) & (_level(pa, pb, na, nb) <= level)
        a, b = torch.cat([a, pa[ok]]), torch.cat([b, pb[ok]])
        uniq, inv = torch.unique(_keys(a, b), return_inverse=True)
        first = torch.full((len(uniq),), len(a), device=DEV).scatter_reduce_(
            0, inv, torch.arange(len(a), device=DEV), "amin").sort().values[:count]
        a, b = a[first], b[first]
        if len(a) == count or len(a) == before:   # complete, or the space is exhausted
            return a, b


def _sd_space(n, ne):
    """HF and all its singles and doubles, as bool[N, n] per spin."""
    hf = torch.zeros(1, n, dtype=torch.bool, device=DEV)
    hf[:, :ne] = True
    ka, kb = _excitations(hf, hf)
    a = torch.cat([hf] + ka)
    b = torch.cat([hf] + kb)
    return a, b


def _excitations(a, b):
    """All singles and doubles of ONE determinant, lists of bool[M, n]."""
    ka, kb = [], []
    one = {}
    for s, X in enumerate((a, b)):
        occ, vir = X[0].nonzero()[:, 0], (~X[0]).nonzero()[:, 0]
        h, p = (t.reshape(-1) for t in torch.meshgrid(occ, vir, indexing="ij"))
        Y = X.repeat(len(h), 1)
        r = torch.arange(len(h), device=DEV)
        Y[r, h] = False
        Y[r, p] = True
        one[s] = Y
        ho, pv = torch.combinations(occ), torch.combinations(vir)
        u, v = (t.reshape(-1) for t in torch.meshgrid(
            torch.arange(len(ho), device=DEV), torch.arange(len(pv), device=DEV), indexing="ij"))
        Z = X.repeat(len(u), 1)
        r = torch.arange(len(u), device=DEV)
        for c in (0, 1):
            Z[r, ho[u, c]] = False
            Z[r, pv[v, c]] = True
        for W in (Y, Z):
            ka.append(W if s == 0 else a.repeat(len(W), 1))
            kb.append(W if s == 1 else b.repeat(len(W), 1))
    u, v = (t.reshape(-1) for t in torch.meshgrid(
        torch.arange(len(one[0]), device=DEV), torch.arange(len(one[1]), device=DEV),
        indexing="ij"))
    ka.append(one[0][u])
    kb.append(one[1][v])
    return ka, kb


def _amplitudes(n, seed):
    """HF-dominated amplitudes with a tail over two decades, normalised."""
    rng = np.random.default_rng(seed + 1)
    x = rng.normal(size=n) * 10.0 ** (-2.0 * rng.random(n))
    x[1:] *= 0.6 / max(np.linalg.norm(x[1:]), 1e-300)
    x[0] = 0.8
    return x


def _system(n, ne, dets, level, seed, space=None):
    h, eri = _integrals(n, seed)
    h1, eri4 = _dense(h, eri, n)
    a, b = _sd_space(n, ne) if space == "sd" else _sample(eri4, n, ne, ne, dets, level, seed + 17)
    return SimpleNamespace(n=n, ne=ne, h=h, eri=eri, h1=h1, eri4=eri4, a=a, b=b)


def _other_phases(s, psi, seed):
    """The same system with other orbital signs, its determinants in another
    order and other amplitude signs: the elements, columns and amplitudes are
    other ones while every |H_ij| and |psi_i|, and so the number of entries
    that screening keeps, stays."""
    rng = np.random.default_rng(seed)
    sg = rng.choice((-1.0, 1.0), s.n)
    i, j = np.tril_indices(s.n)
    pair = torch.from_numpy(sg[i] * sg[j]).to(DEV)
    k, m = torch.tril_indices(len(pair), len(pair), device=DEV)
    s.h = s.h * (sg[i] * sg[j])
    s.eri = s.eri * (pair[k] * pair[m]).cpu().numpy()
    s.h1, s.eri4 = _dense(s.h, s.eri, s.n)
    order = np.concatenate([[0], 1 + rng.permutation(len(psi) - 1)])
    at = torch.from_numpy(order).to(DEV)
    s.a, s.b = s.a[at], s.b[at]
    s.psi = psi[order] * rng.choice((-1.0, 1.0), len(psi))
    return s


#: Kinds whose outputs' sizes depend on the values: one system per case, and
#: _other_phases() of it for each seed.
SIZED_BY_VALUES = ("proxy_eff", "proxy_apply", "conn_amp", "wide_eff", "batch")


def _inputs(case, seed):
    """What a case's prepare() and exact() share."""
    fixed = case["kind"] in SIZED_BY_VALUES
    base = case["dets"] if fixed else seed
    s = _system(case["n_orb"], case["n_el"], case["dets"], case.get("level", 4), base,
                case.get("space"))
    s.psi = _amplitudes(len(s.a), base)
    if case["kind"] == "wide_eff":   # HF and a tail that dynamic screening thins out
        s.psi = np.random.default_rng(base + 1).normal(size=len(s.a)) * 2e-6
        s.psi[0] = 1.0
        s.psi /= np.linalg.norm(s.psi)
    if fixed:
        s = _other_phases(s, s.psi, seed)
    if case["kind"] in ("pt2", "proxy_eff"):   # a reference energy below HF
        s.e_ref = float(_diag(s, s.a[:1], s.b[:1])[0]) - 0.5
    if case["kind"] == "hpsi":
        s.X = np.random.default_rng(seed + 2).normal(size=(len(s.a), case["k"]))
    return s


def _batch_inputs(case, seed):
    rng = np.random.default_rng(case["dets"])
    out = []
    for k in range(case["systems"]):
        n = int(rng.integers(10, 41))
        ne = int(rng.integers(math.ceil(0.4 * n), math.floor(0.6 * n) + 1))
        nd = int(math.exp(rng.uniform(math.log(case["dets"] / 30), math.log(case["dets"]))))
        s = _system(n, ne, nd, 3, case["dets"] + k)
        out.append(_other_phases(s, _amplitudes(len(s.a), case["dets"] + k), seed + k))
    return out


def _bits(n, ne, count, seed):
    """Random determinants around HF: up to 6 excitations, int64[N, 2]."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    out = []
    for _ in range(2):
        # shuffle a few of the orbitals around the Fermi level
        rank = torch.arange(n, device=DEV, dtype=torch.float32).repeat(count, 1)
        far = torch.rand(count, n, generator=g, device=DEV) < 3.0 / n
        rank += far * torch.rand(count, n, generator=g, device=DEV) * (2.0 * ne) * (
            torch.randint(0, 2, (count, n), generator=g, device=DEV) * 2 - 1)
        occ = torch.zeros(count, n, dtype=torch.bool, device=DEV)
        occ.scatter_(1, rank.topk(ne, 1, largest=False).indices, True)
        out.append(_words(occ))
    return torch.cat(out, 1)


def _matrices(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["n"]
    dt = torch.float32 if case["fp32"] else F64
    a = torch.randn(case["batch"], n, n, generator=g, device=DEV, dtype=dt)
    a += n * torch.eye(n, device=DEV, dtype=dt)
    return a, torch.randn(case["batch"], generator=g, device=DEV, dtype=dt)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _precision(case):
    return native.F32 if case.get("fp32") else native.F64


def _context(s, cls=core.IntCtx):
    ctx = cls.from_arrays(s.n, s.h, s.eri, 9.0)
    ctx.hb_prepare()
    return ctx


def prepare(case, seed):
    k = case["kind"]
    st = SimpleNamespace(case=case)
    if k == "features":
        n, ne = case["n_orb"], case["n_el"]
        st.bits = _bits(n, ne, case["dets"], seed)
        st.ref = np.array([(1 << ne) - 1] * 2, dtype=np.uint64)
        st.spec = det_utils.BatchSpec(need_k=True, hp_kmax=case["kmax"], need_phase=case["phase"],
                                      need_hp_pos=case["positions"] and case["kmax"] > 0)
        return st
    if k == "slogdet":
        st.a, st.cot = _matrices(case, seed)
        st.a.requires_grad_(True)
        return st
    if k == "batch":
        ss = _batch_inputs(case, seed)
        st.ctxs = [_context(s) for s in ss]
        st.batch = Batch(st.ctxs, [_masks(s.a, s.b) for s in ss], [s.n for s in ss], eps1=1e-7)
        st.psi = torch.from_numpy(np.concatenate([s.psi for s in ss])).to(DEV)
        st.eloc = torch.empty_like(st.psi)
        return st
    s = _inputs(case, seed)
    st.n = s.n
    st.psi = torch.from_numpy(s.psi).to(DEV)
    if k == "wide_eff":
        st.ctx = _context(s, wide.IntCtxWide)
        st.V = torch.from_numpy(_masks(s.a, s.b, True).view(np.int64)).to(DEV)
        return st
    st.ctx = _context(s)
    st.V_host = _masks(s.a, s.b)
    st.V = torch.from_numpy(st.V_host.view(np.int64)).to(DEV)
    st.system = SimpleNamespace(int_ctx=st.ctx, n_orb=s.n)
    st.space = SimpleNamespace(V_dets=st.V_host)
    st.psi_host = s.psi
    if hasattr(s, "e_ref"):
        st.e_ref = s.e_ref
    if k == "hpsi":
        st.H = device.build(st.ctx, st.V, n_orb=s.n, policy=native.POLICY_STATIC,
                            use_heatbath=True, eps1=1e-6, want_vp=False)
        st.X = torch.from_numpy(s.X).to(DEV)
    if k == "proxy_apply":
        ham, _ = operator.build_proxy_hamiltonian(st.system, st.space, screening="static",
                                                  screen_eps=case["eps1"])
        st.ham = ham
        st.op = operator.build_proxy_operator(ham, precision=_precision(case))
        st.xp = torch.from_numpy(_proxy_amplitudes(len(ham.diagonals.P), seed)).to(DEV)
    return st


def _proxy_amplitudes(n, seed):
    return np.random.default_rng(seed + 3).normal(size=n) / max(n, 1) ** 0.5


def run(st):
    case = st.case
    k = case["kind"]
    if k == "vv_full":
        ham = operator.build_vv_hamiltonian(st.system, st.space)
        e, eloc = operator.local_energy(ham, st.psi)
        return {"e": e, "eloc": eloc, "diag": ham.diagonals.V}
    if k == "vv_static":
        H = device.build(st.ctx, st.V, n_orb=st.n, policy=native.POLICY_STATIC,
                         use_heatbath=True, eps1=case["eps1"], want_vp=False)
        e64, e32 = torch.empty_like(st.psi), torch.empty_like(st.psi)
        s64 = H.local_energy(st.psi, eloc=e64)
        s32 = H.local_energy(st.psi, eloc=e32, precision=native.F32)
        nnz = H.nnz_vv
        H.close()
        return {"eloc64": e64, "eloc32": e32, "sums64": list(s64), "sums32": list(s32),
                "nnz": nnz}
    if k == "hpsi":
        return {"y": st.H.spmv_multi(st.X, precision=_precision(case))}
    if k == "proxy_eff":
        dyn = case["screening"] == "dynamic"
        ham, P = operator.build_proxy_hamiltonian(
            st.system, st.space, screening=case["screening"],
            psi_v=st.psi_host if dyn else None, screen_eps=case["eps1"])
        eff = operator.build_effective_hamiltonian(
            st.system, ham, st.e_ref, epsilon=0.1, precision="fp32" if case["fp32"] else "fp64")
        y = operator.build_vv_operator(eff)(st.psi).V
        return {"y": y, "diag_v": eff.diagonals.V, "diag_p": ham.diagonals.P, "dets_p": P}
    if k == "proxy_apply":
        y = st.op(st.psi, st.xp)
        return {"v": y.V, "p": y.P}
    if k == "conn_amp":
        got = core.get_ham_conn_amp(st.V_host, st.psi_host, st.ctx, st.n, eps1=case["eps1"])
        return {b: {f: got[b][f] for f in ("row", "col", "val")} for b in ("H_VV", "H_VP")} | {
            "det_P": got["det_P"]}
    if k == "energy":
        return {"e": core.compute_variational_energy(st.V, st.psi, st.ctx, st.n,
                                                     use_heatbath=case["heatbath"],
                                                     eps1=case["eps1"])}
    if k == "pt2":
        return core.compute_pt2(st.V, st.psi, st.ctx, st.n, st.e_ref,
                                use_heatbath=case["heatbath"], eps1=case["eps1"])
    if k == "wide_eff":
        H = wide.build_wide(st.ctx, st.V, st.psi, n_orb=st.n, eps1=case["eps1"])
        num, den = H.local_energy(st.psi)
        hpp = torch.empty(H.n_p, dtype=F64, device=DEV)
        wide.p_diag(H, st.ctx, out=hpp)
        eff = wide.ham_eff_wide(H, hpp, num / den, epsilon=0.1, precision=_precision(case))
        y = eff.spmv(st.psi)
        H.close()
        eff.close()
        return {"e_ref": num / den, "diag_p": hpp, "y": y}
    if k == "batch":
        e, _ = st.batch.step(st.psi, precision=_precision(case), graph=True, eloc=st.eloc)
        return {"energies": e, "eloc": st.eloc}
    if k == "features":
        b = det_utils.prepare_batch(st.bits, n_orb=case["n_orb"], n_alpha=case["n_el"],
                                    n_beta=case["n_el"], ref=st.ref, spec=st.spec)
        return {"occ": b.occ, **b.aux}
    if k == "slogdet":
        sign, logabs = slogdet.slogdet_autograd(st.a)
        (grad,) = torch.autograd.grad(logabs, st.a, st.cot)
        return {"sign": sign.detach(), "logabs": logabs.detach(), "grad": grad}
    raise ValueError(f"unknown kind {k}")


# ---------------------------------------------------------------------------
# The work that cannot be left out
# ---------------------------------------------------------------------------

def work(case):
    """Inputs read once, outputs written once; a resident block counts as an
    input of what is applied on it, and an element of a block that a pass
    builds for itself as its arithmetic alone."""
    k, n = case["kind"], case.get("dets", 0)
    if k == "features":
        ne = 2 * case["n_el"]
        row = 16 + 4 * ne + 1 + case["phase"] + case["kmax"] * (9 + 8 * case["positions"])
        return {"bytes": n * row, "flops": 0}
    if k == "slogdet":
        m, size = case["n"], 4 if case["fp32"] else 8
        mats = case["batch"]
        return {"bytes": mats * size * (2 * m * m + 3), "flops": mats * (8 * m ** 3 // 3)}
    if k == "batch":
        n = sum(len(s.a) for s in _batch_inputs(case, 0))
        return {"bytes": 40 * n, "flops": 0}
    if k == "hpsi":
        st = prepare(case, 0)
        n, nnz, kv = st.H.n_v, st.H.nnz_vv, case["k"]
        return {"bytes": nnz * (8 if case["fp32"] else 12) + 16 * n + 16 * n * kv,
                "flops": 2 * nnz * kv}
    if k == "proxy_apply":
        st = prepare(case, 0)
        H = st.ham.ham_vv.device_hamiltonian
        return {"bytes": 12 * (H.nnz_vv + 2 * H.nnz_vp) + 24 * (H.n_v + H.n_p),
                "flops": 2 * (H.nnz_vv + 2 * H.nnz_vp)}
    if k in ("proxy_eff", "conn_amp", "wide_eff"):
        st = prepare(case, 0)
        if k == "wide_eff":
            H = wide.build_wide(st.ctx, st.V, st.psi, n_orb=st.n, eps1=case["eps1"])
        else:
            dyn = case.get("screening") != "static"
            H = device.build(st.ctx, st.V, n_orb=st.n, use_heatbath=True, eps1=case["eps1"],
                             policy=native.POLICY_DYNAMIC if dyn else native.POLICY_STATIC,
                             psi=st.psi if dyn else None)
        io = 32 * H.n_v + (24 if k != "wide_eff" else 8) * H.n_p
        if k == "conn_amp":
            io += 16 * (H.nnz_vv + H.nnz_vp)
        return {"bytes": io, "flops": 2 * (H.nnz_vv + H.nnz_vp)}
    return {"bytes": 24 * n + {"vv_full": 16, "vv_static": 16}.get(k, 0) * n, "flops": 0}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits, from plain torch
# ---------------------------------------------------------------------------

def _diag(s, a, b):
    """<x|H|x> of bool occupations."""
    fa, fb = a.to(F64), b.to(F64)
    J = torch.einsum("ppqq->pq", s.eri4)
    JK = J - torch.einsum("pqqp->pq", s.eri4)
    one = (fa + fb) @ torch.diagonal(s.h1)
    two = 0.5 * (((fa @ JK) * fa).sum(1) + ((fb @ JK) * fb).sum(1)) + ((fa @ J) * fb).sum(1)
    return one + two


def _between(cum, x, y):
    """Parity of the occupied orbitals strictly between x and y, from the
    running counts cum[:, k] = occupied below k."""
    lo, hi = torch.minimum(x, y), torch.maximum(x, y)
    r = torch.arange(len(x), device=DEV)
    return (cum[r, hi] - cum[r, lo + 1]) & 1


def _cum(X):
    c = torch.zeros(X.shape[0], X.shape[1] + 1, dtype=I64, device=DEV)
    c[:, 1:] = X.cumsum(1)
    return c


def _singles_values(s, same, other, h, p):
    """Elements of h -> p in the spin string `same` (rows paired)."""
    J = torch.einsum("hpkk->hpk", s.eri4)
    K = torch.einsum("hkkp->hpk", s.eri4)
    v = s.h1[h, p] + ((J - K)[h, p] * same.to(F64)).sum(1) + (J[h, p] * other.to(F64)).sum(1)
    return torch.where(_between(_cum(same), h, p) == 1, -v, v)


def _same_values(s, X, h1, h2, p1, p2):
    """Elements of h1 -> p1, h2 -> p2 in one spin string."""
    v = s.eri4[h1, p1, h2, p2] - s.eri4[h1, p2, h2, p1]
    par = _between(_cum(X), h1, p1)
    Y = X.clone()
    r = torch.arange(len(h1), device=DEV)
    Y[r, h1] = False
    Y[r, p1] = True
    par = par ^ _between(_cum(Y), h2, p2)
    return torch.where(par == 1, -v, v)


def _pair_values(s, i, j):
    """H of the row pairs (i, j) of a space, all within two excitations and
    i != j, and whether each is a single."""
    v = torch.zeros(len(i), dtype=F64, device=DEV)
    single = torch.zeros(len(i), dtype=torch.bool, device=DEV)
    X, Y = (s.a[i], s.b[i]), (s.a[j], s.b[j])
    deg = [(X[t] & ~Y[t]).sum(1) for t in (0, 1)]
    ends = {}
    for t in (0, 1):
        hole, part = X[t] & ~Y[t], Y[t] & ~X[t]
        lo = lambda m: m.to(torch.int8).argmax(1)                                # noqa: E731
        hi = lambda m: m.shape[1] - 1 - m.flip(1).to(torch.int8).argmax(1)       # noqa: E731
        ends[t] = (lo(hole), hi(hole), lo(part), hi(part))
    for t in (0, 1):
        m = ((deg[t] == 1) & (deg[1 - t] == 0)).nonzero()[:, 0]
        v[m] = _singles_values(s, X[t][m], X[1 - t][m], ends[t][0][m], ends[t][2][m])
        single[m] = True
        m = (deg[t] == 2).nonzero()[:, 0]
        v[m] = _same_values(s, X[t][m], *(e[m] for e in ends[t]))
    m = ((deg[0] == 1) & (deg[1] == 1)).nonzero()[:, 0]
    (ha, _, pa, _), (hb, _, pb, _) = ends[0], ends[1]
    w = s.eri4[ha[m], pa[m], hb[m], pb[m]]
    par = _between(_cum(X[0][m]), ha[m], pa[m]) ^ _between(_cum(X[1][m]), hb[m], pb[m])
    v[m] = torch.where(par == 1, -w, w)
    return v, single


def _connected(s):
    """(i, j, value, single) of all connected row pairs i != j of the space."""
    fa, fb = s.a.to(torch.float32), s.b.to(torch.float32)
    N, out = len(fa), []
    step = max(1, int(2e8) // N)
    for r0 in range(0, N, step):
        common = fa[r0:r0 + step] @ fa.T + fb[r0:r0 + step] @ fb.T
        i, j = (common >= 2 * s.ne - 2.5).nonzero(as_tuple=True)
        i = i + r0
        keep = i != j
        i, j = i[keep], j[keep]
        for q in range(0, len(i), 1 << 22):
            ii, jj = i[q:q + (1 << 22)], j[q:q + (1 << 22)]
            out.append((ii, jj, *_pair_values(s, ii, jj)))
    return [torch.cat(x) for x in zip(*out)]


def _screen(v, single, psi_row, how, eps1):
    """The builders' screening: 'full' keeps all, 'static' heat-bath doubles,
    'dynamic' doubles and singles weighted by the row's amplitude, 'energy'
    the matrix-free contraction's."""
    av = v.abs()
    keep = av > 1e-15
    if how == "static":
        keep &= single | (av >= eps1)
    elif how == "energy":
        keep &= torch.where(single, av > eps1, av >= eps1)
    elif how == "dynamic":
        amp = psi_row.abs()
        keep &= torch.where(single, av * amp >= eps1, av >= eps1 / amp.clamp(min=1e-12))
    return keep


def _vv(s, how, eps1=0.0, psi=None):
    """(i, j, v) of the off-diagonal H_VV entries, and its diagonal."""
    i, j, v, single = _connected(s)
    keep = _screen(v, single, psi[i] if psi is not None else None, how, eps1)
    return (i[keep], j[keep], v[keep]), _diag(s, s.a, s.b)


def _times(n, entries, x):
    i, j, v = entries
    return torch.zeros((n,) + x.shape[1:], dtype=F64, device=DEV).index_add_(
        0, i, v.view(-1, *[1] * (x.dim() - 1)) * x[j])


def _all_excitations(s, psi, how, eps1, limit=1 << 22):
    """(row, a, b, value) of every screened single and double of every row:
    bool kets.  `how` as in _screen, or 'pt2': |v psi_row| >= eps1."""
    n, ne = s.n, s.ne
    N = len(s.a)
    occ = [X.nonzero()[:, 1].view(N, ne) for X in (s.a, s.b)]
    vir = [(~X).nonzero()[:, 1].view(N, n - ne) for X in (s.a, s.b)]
    nv = n - ne
    grid = lambda *m: [t.reshape(-1) for t in torch.meshgrid(                    # noqa: E731
        *(torch.arange(q, device=DEV) for q in m), indexing="ij")]
    ho = torch.combinations(torch.arange(ne, device=DEV))
    pv = torch.combinations(torch.arange(nv, device=DEV))
    out = []

    def keep(r, v, single, flips):
        if how == "pt2":
            k = (v.abs() > 1e-15) & ((v * psi[r]).abs() >= eps1)
        else:
            k = _screen(v, torch.full_like(v, single, dtype=torch.bool),
                        psi[r] if psi is not None else None, how, eps1)
        r, v = r[k], v[k]
        ka, kb = s.a[r], s.b[r]
        q = torch.arange(len(r), device=DEV)
        for X, sp in ((ka, 0), (kb, 1)):
            for h, p in flips[sp]:
                X[q, h[k]] = False
                X[q, p[k]] = True
        out.append((r, ka, kb, v))

    def rows(per):
        step = max(1, limit // max(per, 1))
        for r0 in range(0, N, step):
            yield torch.arange(r0, min(N, r0 + step), device=DEV)

    def spread(R, m):
        return R.repeat_interleave(m), torch.arange(m, device=DEV).repeat(len(R))

    hs, ps = grid(ne, nv)
    hp, pp = grid(len(ho), len(pv))
    for t, (X, O) in enumerate(((s.a, s.b), (s.b, s.a))):
        for R in rows(len(hs)):
            r, c = spread(R, len(hs))
            h, p = occ[t][r, hs[c]], vir[t][r, ps[c]]
            keep(r, _singles_values(s, X[r], O[r], h, p), True,
                 {t: [(h, p)], 1 - t: []})
        for R in rows(len(hp)) if len(hp) else ():
            r, c = spread(R, len(hp))
            h1, h2 = (occ[t][r, ho[hp[c], q]] for q in (0, 1))
            p1, p2 = (vir[t][r, pv[pp[c], q]] for q in (0, 1))
            keep(r, _same_values(s, X[r], h1, h2, p1, p2), False,
                 {t: [(h1, p1), (h2, p2)], 1 - t: []})
    ha, pa, hb, pb = grid(ne, nv, ne, nv)
    for R in rows(len(ha)):
        r, c = spread(R, len(ha))
        i, p = occ[0][r, ha[c]], vir[0][r, pa[c]]
        j, q = occ[1][r, hb[c]], vir[1][r, pb[c]]
        v = s.eri4[i, p, j, q]
        par = _between(_cum(s.a[r]), i, p) ^ _between(_cum(s.b[r]), j, q)
        keep(r, torch.where(par == 1, -v, v), False, {0: [(i, p)], 1: [(j, q)]})
    return [torch.cat(x) for x in zip(*out)]


def _vp(s, psi, how, eps1):
    """Entries (i, k, v) of H_VP and the P occupations, P in (alpha, beta)
    order (n_orb <= 31: one integer orders both strings)."""
    r, ka, kb, v = _all_excitations(s, psi, how, eps1)
    key = (_words(ka)[:, 0] << s.n) | _words(kb)[:, 0]
    mine = (_words(s.a)[:, 0] << s.n) | _words(s.b)[:, 0]
    out = ~torch.isin(key, mine)
    r, ka, kb, v, key = r[out], ka[out], kb[out], v[out], key[out]
    uniq, inv = torch.unique(key, return_inverse=True)
    at = torch.zeros(len(uniq), dtype=I64, device=DEV).scatter_(
        0, inv, torch.arange(len(key), device=DEV))
    return (r, inv, v), ka[at], kb[at]


def exact(case, seed):
    k = case["kind"]
    if k == "wide_eff" or k == "features" or case.get("dets", 0) > 60_000:
        # a list of millions of kets per row, whole numbers only, or too many pairs
        return None
    if k == "slogdet":
        a, cot = _matrices(case, seed)
        a, cot = a.to(F64), cot.to(F64)
        sign, logabs = torch.linalg.slogdet(a)
        grad = cot[:, None, None] * torch.linalg.inv(a).transpose(1, 2)
        return {"sign": sign, "logabs": logabs, "grad": grad}
    if k == "batch":
        e, eloc = [], []
        for s in _batch_inputs(case, seed):
            ent, d = _vv(s, "static", 1e-7)
            x = torch.from_numpy(s.psi).to(DEV)
            y = _times(len(x), ent, x) + d * x
            e.append(torch.stack([x @ y, x @ x]))
            eloc.append(y / x)
        return {"energies": torch.stack(e).cpu().numpy(), "eloc": torch.cat(eloc)}
    s = _inputs(case, seed)
    x = torch.from_numpy(s.psi).to(DEV)
    n = len(x)
    if k in ("vv_full", "vv_static"):
        ent, d = _vv(s, "full" if k == "vv_full" else "static", case.get("eps1", 0.0))
        y = _times(n, ent, x) + d * x
        if k == "vv_full":
            return {"e": float((x @ y) / (x @ x)), "eloc": y / x, "diag": d}
        sums = [float(x @ y), float(x @ x)]
        return {"eloc64": y / x, "eloc32": y / x, "sums64": sums, "sums32": sums, "nnz": None}
    if k == "hpsi":
        ent, d = _vv(s, "static", 1e-6)
        X = torch.from_numpy(s.X).to(DEV)
        return {"y": _times(n, ent, X) + d[:, None] * X}
    if k == "energy":
        ent, d = _vv(s, "energy" if case["heatbath"] else "full", case["eps1"])
        row = x * x >= 1e-12
        y = _times(n, ent, x) + d * x
        return {"e": float((x * y)[row].sum())}
    if k == "pt2":
        ent, d = _vv(s, "full")
        sigma = torch.where(x * x >= 1e-12, _times(n, ent, x) + d * x, 0.0)
        res = (sigma - s.e_ref * x) ** 2 / (s.e_ref - d)
        r, ka, kb, v = _all_excitations(s, x, "pt2", case["eps1"])
        key = (_words(ka)[:, 0] << s.n) | _words(kb)[:, 0]
        out = ~torch.isin(key, (_words(s.a)[:, 0] << s.n) | _words(s.b)[:, 0])
        r, ka, kb, v = r[out], ka[out], kb[out], v[out]
        uniq, inv = torch.unique(key[out], return_inverse=True)
        amp = torch.zeros(len(uniq), dtype=F64, device=DEV).index_add_(0, inv, v * x[r])
        at = torch.zeros(len(uniq), dtype=I64, device=DEV).scatter_(
            0, inv, torch.arange(len(inv), device=DEV))
        hpp = _diag(s, ka[at], kb[at])
        return {"e_pt2_internal": float(res[x * x >= 1e-15].sum()),
                "e_pt2_external": float((amp * amp / (s.e_ref - hpp)).sum()), "n_ext": None}
    how = case.get("screening", "static" if k == "proxy_apply" else "dynamic")
    amp = x if how == "dynamic" else None
    vv, d = _vv(s, how, case["eps1"], amp)
    vp, pa, pb = _vp(s, amp, how, case["eps1"])
    dp = _diag(s, pa, pb)
    vi, vk, vval = vp
    if k == "proxy_apply":
        xp = torch.from_numpy(_proxy_amplitudes(len(dp), seed)).to(DEV)
        return {"v": _times(n, vv, x) + d * x + _times(n, vp, xp),
                "p": _times(len(dp), (vk, vi, vval), x) + dp * xp}
    if k == "conn_amp":
        def ordered(i, j, v):
            return v[torch.argsort(i * (max(len(dp), n) + 1) + j)].cpu().numpy()
        r = torch.arange(n, device=DEV)
        return {"H_VV": {"row": None, "col": None,
                         "val": ordered(torch.cat([vv[0], r]), torch.cat([vv[1], r]),
                                        torch.cat([vv[2], d]))},
                "H_VP": {"row": None, "col": None, "val": ordered(vi, vk, vval)}, "det_P": None}
    den = s.e_ref - dp
    inv = den / (den * den + 0.1 * 0.1)
    z = _times(len(dp), (vk, vi, vval), x) * inv
    diag_eff = d + torch.zeros(n, dtype=F64, device=DEV).index_add_(0, vi, vval ** 2 * inv[vk])
    return {"y": _times(n, vv, x) + d * x + _times(n, vp, z), "diag_v": diag_eff.cpu().numpy(),
            "diag_p": dp.cpu().numpy(), "dets_p": None}
