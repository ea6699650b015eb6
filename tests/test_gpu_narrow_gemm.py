"""Products of one to four columns and batches of single rows: every type and layout at the sizes where a row's pieces, a team of
lanes or a block ends, against plain torch in 64 bits."""
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    return ops, capi


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(128, 1, 8), (50000, 1, 40), (129, 2, 80), (4097, 3, 512), (300, 4, 128), (70000, 1, 256), (1000, 2, 1024),
                                   (127, 2, 64), (500, 5, 64), (500, 1, 36)])
@pytest.mark.parametrize("trans_b", [False, True])
def test_narrow_products(dtype, M, N, K, trans_b):
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(M)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A = r(2, M, K + 8).to(dtype)
    B = r(2, *((N, K) if trans_b else (K, N))).to(dtype)
    bias, slope = r(2, N), torch.rand((2, N), generator=g, device="cuda")
    for out in {dtype, torch.float32}:
        Y = torch.full((2, M, N + 1), 9.0, dtype=out, device="cuda")
        ops.gemm(A, B, Y=Y, bias=bias, bias_kind=capi.XB_BIAS_ROW, trans_b=trans_b, batch=2, M=M, N=N, K=K, lda=K + 8,
                 ldb=B.shape[-1], ldy=N + 1, strides=(M * (K + 8), N * K, N, M * (N + 1)), epilogue=capi.XB_EPI_PRELU,
                 ep=(slope, None, None), ep_count=N, stride_ep=N)
        a, w = A[:, :, :K].double(), (B.transpose(1, 2) if trans_b else B).double()
        want = a @ w + bias.double()[:, None]
        want = torch.where(want < 0, want * slope.double()[:, None], want)
        mag = a.abs() @ w.abs() + bias.double().abs()[:, None]
        # fp32 sums of K products in any order (tensor cores: not every partial sum rounded), then the result's own rounding
        eps = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[out]
        assert ((Y[:, :, :N].double() - want).abs() <= 2 * (K + 2) * 2.0 ** -24 * mag + eps * want.abs()).all()
        assert (Y[:, :, N] == 9.0).all()


@pytest.mark.parametrize("P,N,K", [(500, 36, 100), (32, 4, 1), (33, 256, 256), (31, 36, 100), (64, 60, 33), (40, 37, 20), (70, 16, 4096)])
@pytest.mark.parametrize("epi", ["none", "sigmoid"])
def test_batches_of_single_rows(P, N, K, epi):
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, B, full = r(P, 1, K), r(P, K, N) / K ** 0.5, r(P, 1, N)
    Y = torch.full((P, N + 3), 9.0, device="cuda")
    ops.gemm(A, B, Y=Y, bias=full, bias_kind=capi.XB_BIAS_FULL, batch=P, M=1, N=N, K=K, lda=K, ldb=N, ldy=N, ldbias=N,
             strides=(K, K * N, N, N + 3), alpha=0.5, beta=2.0, epilogue=capi.XB_EPI_SIGMOID if epi == "sigmoid" else 0)
    want = 0.5 * (A.double() @ B.double())[:, 0] + 2 * full.double()[:, 0]
    mag = 0.5 * (A.double().abs() @ B.double().abs())[:, 0] + 2 * full.double().abs()[:, 0]
    tol = (K + 4) * 2.0 ** -24 * mag
    if epi == "sigmoid":
        want, tol = want.sigmoid(), tol + 2.0 ** -20            # __expf and the division
    assert ((Y[:, :N].double() - want).abs() <= tol).all() and (Y[:, N:] == 9.0).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_the_named_engine_keeps_its_order_of_sums(dtype):
    """XB_GEMM_SIMT adds k ascending whatever the number of rows or batches: a row has the bits that it has in a smaller call."""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)
    kw = dict(out_dtype=torch.float32, engine=capi.XB_GEMM_SIMT)
    for N in (1, 2, 4):
        A, B = r(1000, 512), r(512, N)
        few = torch.cat([ops.gemm(A[i:i + 100], B, **kw) for i in range(0, 1000, 100)])
        for M in (127, 128, 1000):
            assert torch.equal(ops.gemm(A[:M], B, **kw), few[:M])
    A, B = r(64, 1, 300), r(64, 300, 36)
    one = torch.stack([ops.gemm(A[i], B[i], **kw) for i in range(64)])
    for P in (31, 32, 64):
        assert torch.equal(ops.gemm(A[:P], B[:P], batch=P, M=1, N=36, K=300, strides=(300, 300 * 36, 0, 36), **kw), one[:P])
