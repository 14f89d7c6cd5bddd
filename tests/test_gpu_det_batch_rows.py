"""Batch features at the edges of a warp's rows, of the staged columns, and
with outputs that are not 16-byte aligned."""

import numpy as np
import pytest

from test_det_batch import random_dets

pytestmark = pytest.mark.gpu


# part-filled warps and blocks; kmax 0, odd, a multiple of 8, at and past the
# 32 columns staged at a time; both string widths
@pytest.mark.parametrize("B", [1, 31, 33, 129])
@pytest.mark.parametrize("n_orb,na,nb,kmax", [(9, 3, 4, 0), (12, 5, 5, 5), (32, 16, 15, 8),
                                              (33, 9, 12, 31), (40, 20, 17, 32), (64, 33, 31, 33)])
def test_edges(port, B, n_orb, na, nb, kmax):
    from detnqs_b200 import core
    rng = np.random.default_rng(B + 7 * n_orb)
    r = random_dets(rng, n_orb, na, nb, 1)[0]
    d = random_dets(rng, n_orb, na, nb, B)
    got = core.prepare_det_batch(d, r, n_orb, na, nb, kmax, True, True, True, kmax > 0)
    want = port.prepare_det_batch(d, r, n_orb, na, nb, kmax, True, True, True, kmax > 0)
    assert set(got) == set(want)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


def test_unaligned_buffers(port):
    """Device determinants and outputs 4 or 8 bytes past a 16-byte boundary,
    through the C ABI."""
    import torch
    from detnqs_b200 import native as N
    rng = np.random.default_rng(3)
    B, n, na, nb, kmax = 70, 30, 12, 11, 8
    r = random_dets(rng, n, na, nb, 1)[0]
    d = random_dets(rng, n, na, nb, B)
    want = port.prepare_det_batch(d, r, n, na, nb, kmax, True, True, True, True)
    raw = torch.zeros(2 * B + 1, dtype=torch.int64, device="cuda")
    raw[1:] = torch.from_numpy(d.view(np.int64).reshape(-1)).cuda()
    i32 = {k: torch.zeros(1 + B * w, dtype=torch.int32, device="cuda")
           for k, w in (("occ", na + nb), ("holes", kmax), ("parts", kmax), ("holes_pos", kmax),
                        ("parts_pos", kmax))}
    i8 = {k: torch.zeros(1 + B * w, dtype=torch.int8, device="cuda")
          for k, w in (("k", 1), ("phase", 1), ("hp_mask", kmax))}
    p = {k: t[1:].data_ptr() for k, t in {**i32, **i8}.items()}
    ref = np.ascontiguousarray(r, np.uint64)
    N.check(N.lib.dnq_prepare_det_batch(raw[1:].data_ptr(), B, ref.ctypes.data, n, na, nb, kmax,
                                        15, p["occ"], p["k"], p["phase"], p["holes"], p["parts"],
                                        p["hp_mask"], p["holes_pos"], p["parts_pos"], 0, None))
    for k, t in {**i32, **i8}.items():
        np.testing.assert_array_equal(t[1:].cpu().numpy().reshape(want[k].shape),
                                      want[k].astype(np.int32), err_msg=k)
        assert int(t[0]) == 0
