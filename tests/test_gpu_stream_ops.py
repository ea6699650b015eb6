"""Stand-alone operators at the sizes where a vector access, a merged axis or a warp's row ends."""
import ctypes as C

import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _L():
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    return capi, ops, capi.lib()


@pytest.mark.parametrize("n,c", [(1, 16), (5, 17), (70, 64), (33, 65), (9, 100), (3, 128), (4, 129), (2, 256), (6, 257), (7, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_softmax_rows(n, c, dtype):
    capi, ops, L = _L()
    x = (torch.randn((n, c), generator=torch.Generator().manual_seed(c)) * 3).to(dtype).cuda()
    x[0, c // 2] = float("-inf")
    y = torch.full_like(x, 7.0)
    capi.check(L.xb_softmax(ops.ptr(x), ops.ptr(y), n, c, 1, ops.dt(x), ops.stream()))
    want = x.double().softmax(1)
    # __expf: 2 ulp + 2^-21 * |x| of its argument's rounding, |x| <= 30; sum and division a few ulp; then the type's half-ulp
    tol = 2.0 ** -15 if dtype == torch.float32 else 2.0 ** -10
    assert ((y.double() - want).abs() <= tol * want + 1e-7).all()
    capi.check(L.xb_softmax(ops.ptr(x), ops.ptr(x), n, c, 1, ops.dt(x), ops.stream()))       # in place
    assert torch.equal(x, y)


def _strides(t, shape):
    """element strides of t broadcast to shape (4 axes)"""
    return (C.c_int64 * 4)(*[0 if t.shape[i] == 1 and shape[i] != 1 else t.stride(i) for i in range(4)])


@pytest.mark.parametrize("op,ref", [(0, torch.add), (1, torch.sub), (2, torch.mul), (3, torch.div), (4, torch.maximum), (5, torch.minimum)])
@pytest.mark.parametrize("a,b,off", [
    ((1, 5, 7, 36), (1, 5, 7, 36), 0), ((3, 5, 1, 36), (1, 1, 7, 36), 0), ((3, 5, 7, 36), (3, 5, 7, 1), 0),
    ((3, 1, 7, 8), (1, 5, 1, 1), 0), ((2, 3, 4, 5), (2, 3, 4, 5), 0), ((2, 3, 4, 6), (1, 1, 1, 6), 0), ((1, 1, 9, 4), (1, 1, 1, 1), 0),
    ((1, 5, 7, 36), (1, 5, 7, 36), 1), ((4, 3, 1, 1), (4, 1, 1, 1), 0)])
def test_elementwise_layouts(op, ref, a, b, off):
    """whole, repeated and merged axes; extents that are no multiple of four; a base that is not 16-byte aligned"""
    capi, ops, L = _L()
    g = torch.Generator().manual_seed(op)
    mk = lambda s: torch.cat([torch.zeros(off), torch.randn(int(np.prod(s)), generator=g) + 2]).cuda()[off:].view(s)
    x, y = mk(a), mk(b)
    shape = torch.broadcast_shapes(a, b)
    out = torch.full(shape, 9.0, device="cuda")
    sh = (C.c_int64 * 4)(*shape)
    names = [capi_op for capi_op in ("XB_EW_ADD", "XB_EW_SUB", "XB_EW_MUL", "XB_EW_DIV", "XB_EW_MAX", "XB_EW_MIN")]
    code = getattr(capi, names[op], op)
    capi.check(L.xb_elementwise(code, ops.ptr(x), _strides(x, shape), ops.ptr(y), _strides(y, shape), None, None, ops.ptr(out),
                                sh, capi.XB_F32, ops.stream()))
    want = ref(x, y).expand(shape)
    assert torch.allclose(out, want, rtol=2.0 ** -22, atol=0)


@pytest.mark.parametrize("rows,cols,src_ld,dst_ld,so,do", [
    (50, 36, 36, 144, 0, 36), (3, 8, 8, 8, 0, 0), (5, 7, 9, 11, 1, 2), (64, 18, 18, 36, 0, 18), (17, 10, 0, 10, 0, 0), (1, 1, 1, 1, 3, 5), (9, 100, 100, 100, 0, 0), (9, 12, 16, 20, 4, 8)])
@pytest.mark.parametrize("dtype,to", [("f32", "f32"), ("f16", "f16"), ("f32", "f16"), ("f16", "f32"), ("i32", "i32"), ("i64", "i64")])
def test_copy2d_pieces(rows, cols, src_ld, dst_ld, so, do, dtype, to):
    capi, ops, L = _L()
    T = dict(f32=torch.float32, f16=torch.float16, i32=torch.int32, i64=torch.int64)
    code = dict(f32=capi.XB_F32, f16=capi.XB_F16, i32=capi.XB_I32, i64=capi.XB_I64)
    src = (torch.arange(so + rows * max(src_ld, cols) + 16) % 1000).to(T[dtype]).cuda()
    dst = torch.full((do + rows * dst_ld + 16,), 5, dtype=T[to], device="cuda")
    want = dst.clone()
    for r in range(rows):
        want[do + r * dst_ld: do + r * dst_ld + cols] = src[so + r * src_ld: so + r * src_ld + cols].to(T[to])
    es = lambda t: t.element_size()
    capi.check(L.xb_copy2d(C.c_void_p(src.data_ptr() + so * es(src)), src_ld, code[dtype], C.c_void_p(dst.data_ptr() + do * es(dst)),
                           dst_ld, code[to], rows, cols, ops.stream()))
    assert torch.equal(dst, want)


@pytest.mark.parametrize("d,du,pad", [(36, 144, 4), (32, 8, 0), (18, 18, 2), (5, 3, 1)])
def test_tower_input_columns(d, du, pad):
    """eight-byte, four-byte and single-element forms of the feature assembly"""
    capi, ops, L = _L()
    R, n, T = 2, 70, 11
    h = lambda *s: torch.randn(s, generator=torch.Generator().manual_seed(d + s[0])).half().cuda()
    user, q, k, att = h(R, du), h(R * n, d), h(R * T, d), h(R * n, d)
    ldx = du + 5 * d + pad
    X = torch.full((R * n, ldx), 9.0, dtype=torch.float16, device="cuda")
    capi.check(L.xb_din_tower_input(ops.ptr(user), du, ops.ptr(q), d, ops.ptr(k), d, ops.ptr(att), d, ops.ptr(X), ldx, R, n, T, d, du,
                                    ops.stream()))
    w = lambda t: t.double().repeat_interleave(n, 0)
    his = w(k.view(R, T, d).double().sum(1))
    q64 = q.double()
    want = torch.cat([w(user), q64, his, q64 * his, att.double(), q64 - his, torch.zeros((R * n, pad), device="cuda", dtype=torch.float64)], 1)
    assert ((X.double() - want).abs() <= 2.0 ** -10 * want.abs() + 2.0 ** -14).all()
