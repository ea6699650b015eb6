"""The extension module's calls hand the C ABI what ops.gemm, PoolPlan.run and Predictor.feed were given: every form of bias,
strides and activation parameters, arrays of every layout, results and exceptions. The C functions are Python callbacks here, so
nothing runs on a GPU."""
import ctypes as C

import numpy as np
import pytest
import torch

import pkg


@pytest.fixture
def bound(monkeypatch):
    pkg.load()
    from x_deeplearning_b200 import blaze_api, capi, ops
    m, seen, result = capi.binding(), [], [0]

    def gemm(a, s):
        seen.append(({n: getattr(a.contents, n) for n, _ in capi.GemmArgs._fields_}, s))
        return result[0]

    def pool(groups, n, scratch, nbytes, s):
        seen.append((groups, n, scratch, nbytes, s))
        return result[0]

    def reshape(h, name, shape, n):
        seen.append(("reshape", h, name, [shape[i] for i in range(n)]))
        return result[0]

    def feed(h, name, data, n):
        seen.append(("feed", h, name, C.string_at(data, n) if n else b""))
        return 0

    fs = {"xb_gemm": C.CFUNCTYPE(C.c_int, C.POINTER(capi.GemmArgs), C.c_void_p)(gemm),
          "xb_embedding_pool": C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_int32, C.c_void_p, C.c_size_t, C.c_void_p)(pool),
          "Blaze_PredictorReshapeInput": C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_char_p, C.POINTER(C.c_int), C.c_int)(reshape),
          "Blaze_PredictorFeed": C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_char_p, C.c_void_p, C.c_int)(feed)}
    real = {n: C.cast(getattr(capi.lib() if n.startswith("xb_") else blaze_api.lib(), n), C.c_void_p).value for n in fs}
    blaze_api.feed_call()
    for n, f in fs.items():
        m.bind(n, C.cast(f, C.c_void_p).value)
    monkeypatch.setattr(ops, "raw_stream", lambda: 77)
    yield ops, capi, blaze_api, seen, result
    for n, a in real.items():
        m.bind(n, a)


def test_gemm_arguments(bound):
    ops, capi, _, seen, result = bound
    A, B = torch.zeros((6, 10), dtype=torch.float16), torch.zeros((12, 10), dtype=torch.float16)[:, :8]
    Y = torch.zeros((6, 24))[:, :12]
    ops.gemm(A[:, :8], B, Y=Y, trans_b=True)
    a, s = seen[-1]
    assert s == 77 and (a["M"], a["N"], a["K"], a["trans_a"], a["trans_b"]) == (6, 12, 8, 0, 1)
    assert (a["A"], a["lda"], a["B"], a["ldb"], a["Y"], a["ldy"]) == (A.data_ptr(), 10, B.data_ptr(), 10, Y.data_ptr(), 24)
    assert (a["alpha"], a["beta"], a["batch"], a["ab_dtype"], a["y_dtype"], a["bias"], a["bias_kind"], a["bias_row_group"]) == (
        1.0, 1.0, 1, capi.XB_F16, capi.XB_F32, None, 0, 0)
    assert (a["ep_a"], a["ep_b"], a["ep_c"], a["ep_count"], a["epilogue"], a["engine"]) == (None, None, None, 0, 0, 0)
    # a row bias, activation parameters, an output of the call's own
    b, slope = torch.zeros(12, dtype=torch.bfloat16), torch.zeros(1)
    y = ops.gemm(A[:, :8], B, bias=b, trans_b=True, epilogue=capi.XB_EPI_PRELU, ep=(slope, None, None), ep_count=1, alpha=0.5, beta=2,
                 engine=1, nosqrt=True, stride_ep=3)
    a, _ = seen[-1]
    assert y.shape == (6, 12) and y.dtype == torch.float16 and a["Y"] == y.data_ptr() and a["ldy"] == 12
    assert (a["bias"], a["bias_kind"], a["ldbias"], a["bias_dtype"]) == (b.data_ptr(), capi.XB_BIAS_ROW, 0, capi.XB_BF16)
    assert (a["alpha"], a["beta"], a["ep_a"], a["ep_count"], a["engine"], a["dice_nosqrt"], a["stride_ep"]) == (
        0.5, 2.0, slope.data_ptr(), 1, 1, 1, 3)
    # a full bias by its own strides, then by given ones; batches; transposed A
    f = torch.zeros((6, 20))[:, :12]
    ops.gemm(A[:, :8], B, bias=f, trans_b=True, bias_row_group=4)
    a, _ = seen[-1]
    assert (a["bias_kind"], a["ldbias"], a["bias_row_group"]) == (capi.XB_BIAS_FULL, 20, 4)
    d = [torch.zeros(3) for _ in range(3)]
    y = ops.gemm(A, B, bias=f, bias_kind=capi.XB_BIAS_ROW, ldbias=9, batch=2, strides=(1, 2, 3, 4), M=5, N=3, K=2, lda=21, ldb=22, ep=d,
                 out_dtype=torch.float32)
    a, _ = seen[-1]
    assert y.shape == (2, 5, 3) and (a["M"], a["N"], a["K"], a["lda"], a["ldb"], a["ldy"], a["ldbias"], a["batch"]) == (5, 3, 2, 21, 22, 3, 9, 2)
    assert (a["stride_a"], a["stride_b"], a["stride_bias"], a["stride_y"]) == (1, 2, 3, 4)
    assert [a["ep_a"], a["ep_b"], a["ep_c"]] == [t.data_ptr() for t in d]
    ops.gemm(A, torch.zeros((6, 4), dtype=torch.float16), trans_a=True)
    assert (seen[-1][0]["M"], seen[-1][0]["K"], seen[-1][0]["N"], seen[-1][0]["trans_a"]) == (10, 6, 4, 1)


def test_gemm_takes_any_indexable(bound):
    ops, capi, _, seen, _ = bound
    A, rows = torch.zeros((4, 4)), torch.zeros((3, 4))
    for ep, strides in ((rows, [1, 2, 3, 4]), ([rows[0], None, rows[2]], range(1, 5)), (dict(enumerate(rows)), torch.Size((1, 2, 3, 4, 5)))):
        ops.gemm(A, A, ep=ep, strides=strides)
        a, _ = seen[-1]
        assert [a["ep_a"], a["ep_b"], a["ep_c"]] == [ep[i] if ep[i] is None else ep[i].data_ptr() for i in range(3)]
        assert (a["stride_a"], a["stride_b"], a["stride_y"]) == (1, 2, 4)


def test_gemm_refuses_and_raises(bound):
    ops, capi, _, seen, result = bound
    A = torch.zeros((4, 4))
    for bad in (dict(B=None), dict(B=A, Y=torch.zeros((4, 4), dtype=torch.float64)), dict(B=A, strides=(0, 0)), dict(B=A, ep=(None,)),
                dict(B=A, M="x", N=1, K=1), dict(B=A, alpha="x"), dict(B=A, bias=3)):
        with pytest.raises((AttributeError, KeyError, TypeError, ValueError, IndexError)):
            ops.gemm(A, **bad)
    assert not seen
    result[0] = -1
    with pytest.raises(capi.XbError):
        ops.gemm(A, A)


def test_pool_and_feed_arguments(bound):
    ops, capi, blaze_api, seen, result = bound
    plan = ops.PoolPlan.__new__(ops.PoolPlan)
    plan._calls, plan._pool = [(1000, 3, 2000, 16), (5000, 1, 6000, 1 << 33)], capi.binding().pool
    plan.run()
    assert seen == [(1000, 3, 2000, 16, 77), (5000, 1, 6000, 1 << 33, 77)]
    del seen[:]
    p = blaze_api.Predictor(C.c_void_p(99))
    whole = np.arange(24, dtype=np.int32).reshape(2, 3, 4)
    for a in (whole, whole[:, ::2], whole.T, np.zeros((0, 5), np.float16), np.float32(3.0), np.array([True, False]),
              np.frombuffer(b"abcd", np.uint8)):
        kept = p.feed("user_0.ids", a)
        want = np.ascontiguousarray(a)
        assert seen[-2:] == [("reshape", 99, b"user_0.ids", list(want.shape)), ("feed", 99, b"user_0.ids", want.tobytes())]
        assert np.array_equal(kept, want) and kept.flags.c_contiguous
    del seen[:]
    result[0] = -1
    with pytest.raises(blaze_api.BlazeError):
        p.feed("x", whole)
    assert len(seen) == 1                              # nothing is fed into an input that could not be reshaped


def test_feed_of_a_closed_predictor(bound):
    _, _, blaze_api, seen, _ = bound
    p = blaze_api.Predictor(C.c_void_p(99))
    p.h = None                                         # what close() leaves
    with pytest.raises(blaze_api.BlazeError):
        p.feed("user_0.ids", np.zeros(3, np.float32))
    assert not seen
