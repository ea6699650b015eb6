"""The kernel library loads without a GPU and exports every entry point that
include/xdlb200.h declares (no compute calls here)."""
import ctypes
import os
import re

import pkg

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "xdlb200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(xb_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    m = pkg.load()
    m.build_native()
    L = ctypes.CDLL(m.capi.LIB_PATH)
    names = declared_symbols()
    assert len(names) >= 20
    for n in names:
        assert hasattr(L, n), "libxdlb200.so does not export %s" % n
    # and the Python binding table covers the header
    assert set(names) == set(m.capi.SYMBOLS), set(names) ^ set(m.capi.SYMBOLS)


def test_argument_errors_are_reported_without_a_gpu():
    m = pkg.load()
    L = m.lib()
    assert L.xb_gemm(None, None) == -1
    assert b"null" in L.xb_last_error()
    assert L.xb_table_row_pitch(18, m.capi.XB_F16) == 48
    assert L.xb_table_row_pitch(16, m.capi.XB_F32) == 64


def test_host_index_builder_matches_lookup_rule():
    import numpy as np
    m = pkg.load()
    keys = np.array([5, 1 << 40, -7, 5, 99], np.int64)          # a repeated key keeps its first row
    slots = 16
    sk = np.zeros(slots, np.int64)
    sr = np.zeros(slots, np.int32)
    rc = m.lib().xb_table_build_index_host(keys.ctypes.data, len(keys), slots, sk.ctypes.data, sr.ctypes.data)
    assert rc == 0
    found = {int(k): int(r) for k, r in zip(sk, sr) if r >= 0}
    assert found == {5: 0, 1 << 40: 1, -7: 2, 99: 4}
    assert m.lib().xb_table_build_index_host(keys.ctypes.data, len(keys), 8, sk.ctypes.data, sr.ctypes.data) == -1


def test_uses_tcgen05_answers_what_the_dispatch_does():
    """Host logic alone: products of up to four columns, few outputs, no depth and fp32 results of [K, N] weights go elsewhere."""
    m = pkg.load()
    c = m.capi

    def uses(M=1000, N=64, K=64, y=None, trans_b=1, engine=c.XB_GEMM_AUTO, lda=None):
        a = c.GemmArgs()
        a.M, a.N, a.K, a.trans_b, a.batch, a.engine = M, N, K, trans_b, 1, engine
        a.A = a.B = a.Y = 4096                               # 16-byte aligned; nothing is read
        a.lda, a.ldb, a.ldy = lda or max(K, 8), (K if trans_b else N) or 8, N
        a.ab_dtype, a.y_dtype = c.XB_F16, y or c.XB_F16
        return m.lib().xb_gemm_uses_tcgen05(ctypes.byref(a))
    assert uses() == 1 and uses(trans_b=0) == 1 and uses(y=c.XB_F32) == 1
    assert uses(N=4) == 0 and uses(N=4, lda=72) == 0 and uses(M=100000, N=5) == 1
    assert uses(K=0) == 0 and uses(K=0, engine=c.XB_GEMM_TCGEN05) == 0
    assert uses(M=127) == 0 and uses(M=128) == 1 and uses(M=127, y=c.XB_F32) == 0
    assert uses(y=c.XB_F32, trans_b=0) == 0 and uses(lda=65) == 0
    assert uses(M=127, engine=c.XB_GEMM_TCGEN05) == 1 and uses(trans_b=0, engine=c.XB_GEMM_TCGEN05) == 0
    assert uses(engine=c.XB_GEMM_SIMT) == 0
