"""A call that fails in the CUDA runtime leaves the next one alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_next_call_after_a_runtime_error():
    from detnqs_b200 import core, native as N
    a, b = np.array([[3, 3]], np.uint64), np.array([[5, 3]], np.uint64)
    want = core.excitations(a, b)
    for _ in range(2):
        with pytest.raises(N.DetnqsError, match="invalid device ordinal"):
            core.excitations(a, b, device=99)
        got = core.excitations(a, b)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
