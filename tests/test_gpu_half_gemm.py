"""16-bit products off the tensor-memory path (odd rows, odd starts, transposed A, few outputs): every layout at the edges of the
64-wide tiles and of the 64-deep slices, against plain torch in 64 bits."""
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    return ops, capi


# (off: elements that A starts behind an aligned address; pad: what the rows of A, B and Y have beyond their elements)
@pytest.mark.parametrize("M,N,K,batch,off,pad", [
    (1, 5, 1, 1, 0, 0), (20, 56, 72, 2, 0, 0), (33, 64, 312, 2, 0, 0), (63, 63, 63, 3, 0, 0), (64, 64, 64, 1, 1, 1), (65, 65, 65, 2, 1, 0),
    (127, 31, 16, 1, 0, 1), (128, 66, 15, 2, 2, 2), (129, 129, 17, 1, 1, 0), (300, 7, 313, 1, 0, 0), (2000, 325, 29, 4, 0, 0),
    (10159, 31, 129, 1, 0, 0), (4000, 190, 130, 1, 2, 0), (2500, 511, 500, 1, 0, 0)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_odd_products(M, N, K, batch, off, pad, trans_a, trans_b, dtype):
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    ar, ac = (K, M) if trans_a else (M, K)
    br, bc = (N, K) if trans_b else (K, N)
    lda, ldb, ldy = ac + pad, bc + pad, N + pad
    flat = r(off + batch * ar * lda).to(dtype)
    A, B = flat[off:], r(batch, br, ldb).to(dtype)
    bias, slope = r(batch, N), torch.rand((batch, N), generator=g, device="cuda")
    Y = torch.full((batch, M + 1, ldy), 9.0, dtype=dtype, device="cuda")
    ops.gemm(A, B, Y=Y, bias=bias, bias_kind=capi.XB_BIAS_ROW, trans_a=trans_a, trans_b=trans_b, batch=batch, M=M, N=N, K=K, lda=lda,
             ldb=ldb, ldy=ldy, strides=(ar * lda, br * ldb, N, (M + 1) * ldy), epilogue=capi.XB_EPI_PRELU, ep=(slope, None, None),
             ep_count=N, stride_ep=N)
    a = A.view(batch, ar, lda)[:, :, :ac].double()
    w = B[:, :, :bc].double()
    a, w = a.transpose(1, 2) if trans_a else a, w.transpose(1, 2) if trans_b else w
    want = a @ w + bias.double()[:, None]
    mag = a.abs() @ w.abs() + bias.double().abs()[:, None]
    want = torch.where(want < 0, want * slope.double()[:, None], want)
    # fp32 sums of K products, not every one rounded; then the result's rounding (fp16 below its normal range: half its smallest step)
    eps, tiny = (2.0 ** -11, 2.0 ** -25) if dtype == torch.float16 else (2.0 ** -8, 0.0)
    assert ((Y[:, :M, :N].double() - want).abs() <= 2 * (K + 2) * 2.0 ** -24 * mag + eps * want.abs() + tiny).all()
    assert (Y[:, M:] == 9.0).all() and (Y[:, :, N:] == 9.0).all()


def test_bias_matrix_and_other_activations():
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    M, N, K, group = 150, 67, 45, 7
    A, B, full = r(M, K).half(), (r(K, N) / K ** 0.5).half(), r((M + group - 1) // group, N)
    want = 0.5 * (A.double() @ B.double()) + 2 * full.double().repeat_interleave(group, 0)[:M]
    Y = ops.gemm(A, B, bias=full, bias_kind=capi.XB_BIAS_FULL, bias_row_group=group, alpha=0.5, beta=2.0, epilogue=capi.XB_EPI_SIGMOID)
    assert (Y.double() - want.sigmoid()).abs().max() <= 2.0 ** -12 + (K + 4) * 2.0 ** -22
    gamma, mean, var = torch.rand(N, generator=g, device="cuda"), r(N), torch.rand(N, generator=g, device="cuda") + 0.5
    Y = ops.gemm(A, B, epilogue=capi.XB_EPI_DICE, ep=(gamma, mean, var))
    x = A.double() @ B.double()
    p = ((x - mean.double()) / var.double().sqrt()).sigmoid()
    want = (1 - p) * gamma.double() * x + p * x
    # (|d dice / d x| <= 1 + |x| / 4 std)
    assert ((Y.double() - want).abs() <= 2.0 ** -11 * want.abs() + (K + 4) * 2.0 ** -22 * (1 + x.abs() / 2) * 4).all()


def test_zero_depth_is_the_bias():
    ops, capi = _ops()
    bias = torch.randn(70, device="cuda")
    Y = ops.gemm(torch.empty((40, 1), dtype=torch.float16, device="cuda"), torch.empty((1, 70), dtype=torch.float16, device="cuda"), bias=bias,
                 bias_kind=capi.XB_BIAS_ROW, M=40, N=70, K=0, lda=1, ldb=70)
    assert torch.equal(Y, bias.half().expand(40, 70))


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 8, 8), (3, 2, 17), (1, 5, 64), (2, 16, 65), (16, 1, 200), (127, 3, 8)])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_smallest_aligned_products(M, N, K, trans_b, dtype):
    """(rows at 16-byte addresses: the tensor-memory path from one output on)"""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(K)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    up = lambda n: (n + 7) // 8 * 8
    A, B = r(2, M, up(K)).to(dtype), r(2, *((N, up(K)) if trans_b else (K, up(N)))).to(dtype)
    Y = torch.full((2, M, N + 1), 9.0, dtype=dtype, device="cuda")
    ops.gemm(A, B, Y=Y, trans_b=trans_b, batch=2, M=M, N=N, K=K, lda=up(K), ldb=B.shape[-1], ldy=N + 1,
             strides=(M * up(K), B[0].numel(), 0, M * (N + 1)))
    a = A[:, :, :K].double()
    w = B[:, :, :K].double().transpose(1, 2) if trans_b else B[:, :, :N].double()
    eps, tiny = (2.0 ** -11, 2.0 ** -25) if dtype == torch.float16 else (2.0 ** -8, 0.0)
    assert ((Y[:, :, :N].double() - a @ w).abs() <= 2 * (K + 2) * 2.0 ** -24 * (a.abs() @ w.abs()) + eps * (a @ w).abs() + tiny).all()
    assert (Y[:, :, N] == 9.0).all()


@pytest.mark.parametrize("M,N", [(3000, 257), (70, 33)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("epi", ["sigmoid", "dice"])
def test_activations_as_on_the_cuda_cores(M, N, dtype, epi):
    """Sums that any order leaves exact (one product each): bias and activation give the bits of XB_GEMM_SIMT."""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(M)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, W = torch.zeros((M, 65), dtype=dtype, device="cuda"), r(65, N).to(dtype)
    A[:, 40] = r(M).to(dtype)
    u = lambda lo, hi: torch.rand((N,), generator=g, device="cuda") * (hi - lo) + lo
    kw = dict(epilogue=capi.XB_EPI_SIGMOID) if epi == "sigmoid" else dict(epilogue=capi.XB_EPI_DICE, ep=(u(0, 0.5), u(-0.1, 0.1), u(0.5, 1.5)))
    got, simt = [ops.gemm(A, W, bias=r(N) * 0 + 0.3, engine=e, **kw) for e in (capi.XB_GEMM_AUTO, capi.XB_GEMM_SIMT)]
    assert torch.equal(got, simt)


@pytest.mark.parametrize("M,N,K,batch", [(300, 65, 301, 2), (9000, 65, 129, 1), (60, 64, 320, 1), (22, 16, 512, 16)])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("positive", [False, True])
def test_sums_are_no_worse_than_fp32_fmas(M, N, K, batch, trans_b, dtype, positive):
    """A full bias takes the exact sums away and a factor brings what is left, the errors of the sums, into a 16-bit result."""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(K)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, B = r(batch, M, K), r(batch, *((N, K) if trans_b else (K, N))) / K ** 0.5
    A, B = [(x.abs() if positive else x).to(dtype) for x in (A, B)]
    exact = A.double() @ (B.transpose(1, 2) if trans_b else B).double()
    full, scale = exact.float(), 2.0 ** 20
    rms = []
    for e in (capi.XB_GEMM_AUTO, capi.XB_GEMM_SIMT):
        Y = ops.gemm(A, B, bias=-full, bias_kind=capi.XB_BIAS_FULL, trans_b=trans_b, batch=batch, M=M, N=N, K=K, lda=K, ldb=B.shape[-1], ldy=N,
                     ldbias=N, strides=(M * K, N * K, M * N, M * N), alpha=scale, beta=scale, engine=e,
                     Y=torch.empty((batch, M, N), dtype=dtype, device="cuda"))
        rms.append((Y.double() / scale + (full.double() - exact)).pow(2).mean().sqrt().item())
    assert rms[0] <= rms[1], rms


@pytest.mark.parametrize("M,N,K,batch", [(706, 43, 14, 1), (46002, 15, 16, 1), (42, 119, 7, 1), (1087, 121, 3, 1), (38, 11, 8, 2), (5, 3, 1, 1)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_one_shallow_slice_is_the_cuda_cores(M, N, K, batch, dtype):
    """The low bits of the sums, brought into a 16-bit result as above, are those of XB_GEMM_SIMT."""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(K)
    A, B = [torch.randn(s, generator=g, device="cuda").to(dtype) for s in ((batch, M, K), (batch, K, N))]
    full = -(A.double() @ B.double()).float()
    got = [ops.gemm(A, B, bias=full, bias_kind=capi.XB_BIAS_FULL, batch=batch, M=M, N=N, K=K, lda=K, ldb=N, ldy=N, ldbias=N, alpha=2.0 ** 20,
                    beta=2.0 ** 20, strides=(M * K, K * N, M * N, M * N), engine=e, Y=torch.empty((batch, M, N), dtype=dtype, device="cuda"))
           for e in (capi.XB_GEMM_AUTO, capi.XB_GEMM_SIMT)]
    assert torch.equal(*got)
