"""Electron counts beyond the orbitals: refused like any other mismatch, with
the oracle's message for the first failing determinant, however large."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one spin and both past n_orb; pieces below, at and past a block's shared
# memory (449 electrons), and past 32 bits of bytes
@pytest.mark.parametrize("n_orb,na,nb", [(12, 13, 0), (12, 0, 13), (64, 65, 64), (40, 300, 148),
                                         (40, 300, 150), (64, 1000, 1000), (20, 9_000_000, 3)])
@pytest.mark.parametrize("bad_bits", [False, True])
@pytest.mark.parametrize("hp", [False, True])
def test_counts_past_the_orbitals(port, n_orb, na, nb, bad_bits, hp):
    from detnqs_b200 import core
    if bad_bits and n_orb == 64:
        pytest.skip("64 orbitals take every bit")
    d = np.array([[7, 3]] * 3, np.uint64)
    if bad_bits:
        d[0, 1] |= np.uint64(1) << np.uint64(n_orb)
    args = (d, np.array([7, 7], np.uint64), n_orb, na, nb, 4 if hp else 0, True, False, hp)
    with pytest.raises(ValueError) as want:
        port.prepare_det_batch(*args)
    with pytest.raises(ValueError) as got:
        core.prepare_det_batch(*args)
    assert str(got.value) == str(want.value)
    # and the next call runs
    ok = core.prepare_det_batch(d[1:], np.array([7, 3], np.uint64), 12, 3, 2)
    np.testing.assert_array_equal(ok["occ"], [[0, 1, 2, 12, 13]] * 2)
