"""Downfolding kernel: rows in one unit and in two halves, columns longer than
the list of steps, accumulators in shared and in global memory."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(nv, n_p, per_col, seed):
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for k in range(n_p):
        m = nv if k == 0 else min(nv, int(rng.integers(1, 2 * per_col)))
        rows.append(np.sort(rng.choice(nv, m, replace=False)))
        cols.append(np.full(m, k))
    r, c = np.concatenate(rows).astype(np.uint32), np.concatenate(cols).astype(np.uint32)
    v = rng.normal(size=r.size)
    v[rng.random(r.size) < 0.02] = 0.0            # stored zeros
    order = np.lexsort((c, r))
    vp = {"row": r[order], "col": c[order], "val": v[order], "shape": (nv, n_p)}
    d = rng.integers(0, nv, 3 * nv)
    e = rng.integers(0, nv, 3 * nv)
    key = np.unique(d.astype(np.int64) * nv + e)
    vv = {"row": (key // nv).astype(np.uint32), "col": (key % nv).astype(np.uint32),
          "val": rng.normal(size=key.size), "shape": (nv, nv)}
    hpp = 1.0 + 9.0 * rng.random(n_p)
    return vv, vp, hpp


def _reference(vv, vp, hpp, nv):
    """Terms added one after the other in column order, and their magnitudes."""
    dinv = 1.0 / (0.0 - hpp)
    acc, mag = np.zeros((nv, nv)), np.zeros((nv, nv))
    order = np.argsort(vp["col"], kind="stable")
    r, c, v = vp["row"][order], vp["col"][order], vp["val"][order]
    for k in range(hpp.size):
        lo, hi = np.searchsorted(c, [k, k + 1])
        i, a = r[lo:hi].astype(np.int64), v[lo:hi]
        if abs(dinv[k]) * np.sum(a * a) < 1e-12:
            continue
        t = (a * dinv[k])[:, None] * a[None, :]
        acc[np.ix_(i, i)] += t
        mag[np.ix_(i, i)] += np.abs(t)
    h = np.zeros((nv, nv))
    h[vv["row"], vv["col"]] = vv["val"]
    return h + acc, mag


# one unit a row (below 64 rows or short columns) and two; odd halves; a column
# of more steps than are listed at a time; 6,401 rows: global accumulators
@pytest.mark.parametrize("nv,n_p,per_col", [(63, 90, 30), (64, 90, 30), (65, 200, 40),
                                            (65, 200, 5), (130, 33, 60), (4203, 7, 40),
                                            (6401, 3, 40)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_terms_in_column_order(nv, n_p, per_col, precision):
    from detnqs_b200 import core
    vv, vp, hpp = _blocks(nv, n_p, per_col, nv + n_p)
    got = core.get_ham_eff(vv, vp, hpp, 0.0, reg_type="linear_shift", epsilon=0.0,
                           precision=precision)
    want, mag = _reference(vv, vp, hpp, nv)
    h = np.zeros((nv, nv))
    h[got["row"], got["col"]] = got["val"]
    key = got["row"].astype(np.int64) * nv + got["col"]
    assert np.all(np.diff(key) > 0)
    if precision == "fp64":
        assert np.array_equal(h, np.where(np.abs(want) > 1e-15, want, 0.0))
    else:   # two values rounded to FP32 in each term (2^-24 each)
        assert np.all(np.abs(h - want) <= 1.3e-7 * mag + 1e-15)
