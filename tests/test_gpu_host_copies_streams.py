"""Staged copies to the host behind work on the caller's stream, whatever
handle names it: the default streams, cudaStreamPerThread (another stream in
every thread) and a stream of the caller."""

import ctypes as C

import numpy as np
import pytest

from detnqs_b200 import synthetic as S

pytestmark = pytest.mark.gpu

STREAMS = {"default": lambda: None, "legacy": lambda: 1, "per_thread": lambda: 2}


def _side():
    import torch
    s = torch.cuda.Stream()
    STREAMS["side"].keep = s
    return s.cuda_stream


STREAMS["side"] = _side


@pytest.fixture(scope="module")
def ctx():
    from detnqs_b200 import core
    n = 20
    sysm = S.make_system(n, 7, 7, 2 * n, 5)
    c = core.IntCtx.from_arrays(n, sysm.h1e, sysm.eri, sysm.e_core)
    c.hb_prepare(1e-15)
    yield c
    c.close()


def _build(ctx, V, stream, want_vp):
    from detnqs_b200 import native as N
    h = C.c_void_p()
    N.check(N.lib.dnq_build(ctx.handle, V.ctypes.data, len(V), None, 0, None, 20,
                            N.POLICY_STATIC, 1, 1e-7, want_vp, stream, C.byref(h)))
    info = np.zeros(6, np.int64)
    N.check(N.lib.dnq_ham_info(h, info.ctypes.data))
    return h, info


def _coo(ctx, V, stream, block):
    """A block right after its build (V->V rows are still to be sorted and
    gathered on the stream), and the same through the CSR and P copies."""
    from detnqs_b200 import native as N
    out = []
    h, info = _build(ctx, V, stream, block)
    nnz = int(info[3 if block else 1])
    assert 4 * nnz >= 8 << 20   # every array is staged
    arrays = [np.empty(nnz, np.uint32), np.empty(nnz, np.uint32), np.empty(nnz, np.float64)]
    N.check(N.lib.dnq_ham_copy_coo(h, block, *(a.ctypes.data for a in arrays), stream))
    out += arrays
    N.check(N.lib.dnq_ham_destroy(h))
    h, info = _build(ctx, V, stream, block)
    arrays = [np.empty(len(V) + 1, np.int64), np.empty(nnz, np.uint32), np.empty(nnz, np.float64)]
    N.check(N.lib.dnq_ham_copy_csr(h, block, *(a.ctypes.data for a in arrays), stream))
    out += arrays
    if block:
        assert 16 * info[2] >= 8 << 20
        p = np.empty((int(info[2]), 2), np.uint64)
        N.check(N.lib.dnq_ham_copy_dets_p(h, p.ctypes.data, stream))
        out.append(p)
    N.check(N.lib.dnq_ham_destroy(h))
    return out


@pytest.mark.parametrize("block", [0, 1])
@pytest.mark.parametrize("name", ["legacy", "per_thread", "side"])
def test_blocks(ctx, name, block):
    V = S.hf_sd_space(20, 7, 7)
    V = np.ascontiguousarray(V if block == 0 else V[:600])
    want = _coo(ctx, V, None, block)
    got = _coo(ctx, V, STREAMS[name](), block)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("name", ["legacy", "per_thread", "side"])
def test_connections(ctx, name):
    from detnqs_b200 import native as N
    V = np.ascontiguousarray(S.hf_sd_space(20, 7, 7)[:300])

    def conn(stream):
        h = C.c_void_p()
        N.check(N.lib.dnq_local_connections(ctx.handle, V.ctypes.data, len(V), 20, 1, 1e-7, stream,
                                            C.byref(h)))
        info = np.zeros(6, np.int64)
        N.check(N.lib.dnq_ham_info(h, info.ctypes.data))
        m = int(info[2])
        assert 8 * m >= 8 << 20
        off, d, v = np.empty(len(V) + 1, np.int32), np.empty((m, 2), np.uint64), np.empty(m)
        N.check(N.lib.dnq_conn_copy(h, off.ctypes.data, d.ctypes.data, v.ctypes.data, stream))
        N.check(N.lib.dnq_ham_destroy(h))
        return off, d, v

    for a, b in zip(conn(STREAMS[name]()), conn(None)):
        np.testing.assert_array_equal(a.view(np.uint8), b.view(np.uint8))
