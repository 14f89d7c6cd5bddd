"""A build on a GPU with little memory left, all of it scattered over the
pool's unused pieces: the arena shrinks and the two-pass walk builds the
block."""

import contextlib

import numpy as np
import pytest

from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MB = 1 << 20
LEFT = 192 * MB   # to be left free; the whole arena of this build takes 350 MB


@contextlib.contextmanager
def _full():
    """The device's pool with 15 MB holes (more than an arena in all) between
    pieces in use, and the device filled up to LEFT."""
    rt = pytest.importorskip("cuda.bindings.runtime")

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1] if len(r) > 1 else None

    pool = ok(rt.cudaDeviceGetDefaultMemPool(0))
    ok(rt.cudaDeviceSynchronize())
    ok(rt.cudaMemPoolTrimTo(pool, 0))
    pieces, fill = [], []
    try:
        for _ in range(1024):
            pieces.append(ok(rt.cudaMallocAsync(MB, 0)))
        for p in [p for k, p in enumerate(pieces) if k % 16]:
            pieces.remove(p)
            ok(rt.cudaFreeAsync(p, 0))
        ok(rt.cudaDeviceSynchronize())
        size = 64 << 30
        while size >= 8 * MB:
            free = rt.cudaMemGetInfo()[1]
            if free - size >= LEFT:
                fill.append(ok(rt.cudaMalloc(size)))
            else:
                size //= 2
        yield
    finally:
        for p in fill:
            rt.cudaFree(p)
        for p in pieces:
            rt.cudaFreeAsync(p, 0)
        ok(rt.cudaDeviceSynchronize())
        ok(rt.cudaMemPoolTrimTo(pool, 0))


def test_build_in_scattered_memory():
    from detnqs_b200 import core, device, native as N
    n = 13
    sysm = S.make_system(n, 5, 5, 2 * n, 3)
    V = np.ascontiguousarray(S.hf_sd_space(n, 5, 5)[:2000])
    ctx = core.IntCtx.from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    ctx.hb_prepare(1e-15)

    def block():
        H = device.build(ctx, V, n_orb=n, policy=N.POLICY_STATIC, use_heatbath=True, eps1=1e-6,
                         want_vp=False)
        try:
            return H.to_coo(0)
        finally:
            H.close()

    want = block()
    N.check(N.lib.dnq_set_option(N.OPT_ARENA_CAP, 1024))   # the two-pass kernels load here
    try:
        block()
    finally:
        N.check(N.lib.dnq_set_option(N.OPT_ARENA_CAP, 0))
    with _full():
        got = block()
    for key in ("row", "col", "val"):
        np.testing.assert_array_equal(got[key].view(np.uint8), want[key].view(np.uint8))
    ctx.close()
