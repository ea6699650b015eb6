"""Outputs that end inside a tile, with one tile a block (stored by the threads) and with several (stored by TMA), batches stacked or
side by side, against plain torch in 64 bits; what lies around the output stays as it was."""
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    return ops, capi


EPI = ["none", "prelu", "dice", "sigmoid"]


@pytest.mark.parametrize("N", [8, 16, 24, 40, 64, 72, 104, 128, 136, 144, 152, 168, 200, 256, 264, 272, 328, 392, 600])
@pytest.mark.parametrize("M", [6401, 130])
@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("dtype,out", [(torch.float16, torch.float16), (torch.bfloat16, torch.bfloat16), (torch.float16, torch.float32)])
def test_ragged_outputs(N, M, beside, dtype, out):
    ops, capi = _ops()
    P, K = 3, 72
    kn = N % 16 == 0 and out != torch.float32
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, B = r(P, M, K).to(dtype), (r(P, N, K) / K ** 0.5).to(dtype)
    bias = r(P, N)
    act = EPI[(N // 8 + beside) % 4]
    kw, x = {}, A.double() @ B.double().transpose(1, 2) + bias.double()[:, None]
    mag = A.double().abs() @ B.double().abs().transpose(1, 2) + bias.double().abs()[:, None]
    slope = torch.rand((P, N), generator=g, device="cuda")
    if act == "prelu":
        kw = dict(epilogue=capi.XB_EPI_PRELU, ep=(slope, None, None), ep_count=N, stride_ep=N)
        want = torch.where(x < 0, x * slope.double()[:, None], x)
    elif act == "dice":
        mean, var = r(P, N), torch.rand((P, N), generator=g, device="cuda") + 0.5
        kw = dict(epilogue=capi.XB_EPI_DICE, ep=(slope, mean, var), stride_ep=N)
        p = ((x - mean.double()[:, None]) / var.double().sqrt()[:, None]).sigmoid()
        want = (1 - p) * slope.double()[:, None] * x + p * x
    elif act == "sigmoid":
        kw, want = dict(epilogue=capi.XB_EPI_SIGMOID), x.sigmoid()
    else:
        want = x
    ld = N * P + 16 if beside else N + 8
    Y = torch.full((M + 1, ld) if beside else (P * M + 1, ld), 9.0, dtype=out, device="cuda")
    W = B.transpose(1, 2).contiguous() if kn else B
    ops.gemm(A, W, Y=Y, bias=bias, bias_kind=capi.XB_BIAS_ROW, trans_b=not kn, batch=P, M=M, N=N, K=K, lda=K, ldb=W.shape[-1], ldy=ld,
             strides=(M * K, N * K, N, N if beside else M * ld), **kw)
    got = Y[:M, :P * N].view(M, P, N).transpose(0, 1) if beside else Y[:P * M].view(P, M, ld)[:, :, :N]
    # fp32 sums of K products, not every one rounded; the activations' slopes (Dice: at most 1 + |x| / (2 std)) and their fast
    # exponential and quotient; the result's rounding
    eps = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}[out]
    tol = 2 * (K + 2) * 2.0 ** -24 * mag
    if act == "dice":
        tol = tol * (1 + x.abs()) + 2.0 ** -20 * (1 + x.abs())
    elif act == "sigmoid":
        tol = tol + 2.0 ** -20
    assert ((got.double() - want).abs() <= tol + eps * want.abs() + (2.0 ** -25 if out == torch.float16 else 0)).all()
    if beside:
        assert (Y[M:] == 9.0).all() and (Y[:, P * N:] == 9.0).all()
    else:
        assert (Y[P * M:] == 9.0).all() and (Y[:, N:] == 9.0).all()


@pytest.mark.parametrize("M,N,K,P,beside", [(9700, 512, 392, 1, False), (9700, 256, 640, 2, True), (4990, 512, 384, 2, False), (18945, 256, 400, 1, False)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_two_cta_tiles_end_anywhere(M, N, K, P, beside, dtype):
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, B, bias = r(P, M, K).to(dtype), (r(P, N, K) / K ** 0.5).to(dtype), r(P, N)
    slope = torch.rand((P, N), generator=g, device="cuda")
    ld = N * P + 16 if beside else N + 8
    Y = torch.full((M + 1, ld) if beside else (P * M + 1, ld), 9.0, dtype=dtype, device="cuda")
    ops.gemm(A, B, Y=Y, bias=bias, bias_kind=capi.XB_BIAS_ROW, trans_b=True, batch=P, M=M, N=N, K=K, lda=K, ldb=K, ldy=ld,
             strides=(M * K, N * K, N, N if beside else M * ld), epilogue=capi.XB_EPI_PRELU, ep=(slope, None, None), ep_count=N, stride_ep=N)
    x = A.double() @ B.double().transpose(1, 2) + bias.double()[:, None]
    mag = A.double().abs() @ B.double().abs().transpose(1, 2) + bias.double().abs()[:, None]
    want = torch.where(x < 0, x * slope.double()[:, None], x)
    got = Y[:M, :P * N].view(M, P, N).transpose(0, 1) if beside else Y[:P * M].view(P, M, ld)[:, :, :N]
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert ((got.double() - want).abs() <= 2 * (K + 2) * 2.0 ** -24 * mag + eps * want.abs() + (2.0 ** -25 if dtype == torch.float16 else 0)).all()
    if beside:
        assert (Y[M:] == 9.0).all() and (Y[:, P * N:] == 9.0).all()
    else:
        assert (Y[P * M:] == 9.0).all() and (Y[:, N:] == 9.0).all()


@pytest.mark.parametrize("N", [80, 104, 160, 200, 256, 272])
@pytest.mark.parametrize("M,P,K", [(289, 500, 8), (289, 500, 24), (545, 300, 24), (130, 800, 16)])
def test_ragged_tiles_between_whole_ones(N, M, P, K):
    """Ten and more tiles a block, every third or fifth of them with warps whose rows all lie past the output, stores that the copies
    queue behind: each launch has the bits that the batches have one at a time (one tile a block, stored by the threads)."""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, B, bias = r(P, M, K).half(), (r(P, N, K) / K ** 0.5).half(), r(P, N)
    one = torch.empty((P, M, N), dtype=torch.float16, device="cuda")
    for b in range(P):
        ops.gemm(A[b], B[b], Y=one[b], bias=bias[b], trans_b=True)
    many = [torch.full((P, M, N), 9.0, dtype=torch.float16, device="cuda") for _ in range(4)]
    for Y in many:
        ops.gemm(A, B, Y=Y, bias=bias, bias_kind=capi.XB_BIAS_ROW, trans_b=True, batch=P, M=M, N=N, K=K, lda=K, ldb=K, ldy=N,
                 strides=(M * K, N * K, N, M * N))
    for Y in many:
        assert torch.equal(Y, one)
    x = A.double() @ B.double().transpose(1, 2) + bias.double()[:, None]
    mag = A.double().abs() @ B.double().abs().transpose(1, 2) + bias.double().abs()[:, None]
    # fp32 sums of K products, not every one rounded, and the result's rounding
    assert ((one.double() - x).abs() <= 2 * (K + 2) * 2.0 ** -24 * mag + 2.0 ** -11 * x.abs() + 2.0 ** -25).all()


# (by TMA, in pieces, rows that start anywhere)
@pytest.mark.parametrize("M,N", [(40000, 200), (5000, 200), (20000, 199)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_sigmoid_of_16_bits_is_the_rounding_of_fp32(M, N, dtype):
    """The activation is fp32 arithmetic whatever the result's type: the same product with an fp32 result, rounded."""
    ops, capi = _ops()
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    A, W, bias = r(M, 88).to(dtype), (r(N, 88) / 6).to(dtype), r(N)
    kw = dict(bias=bias, trans_b=True, epilogue=capi.XB_EPI_SIGMOID, engine=capi.XB_GEMM_TCGEN05)
    got, fp32 = ops.gemm(A, W, out_dtype=dtype, **kw), ops.gemm(A, W, out_dtype=torch.float32, **kw)
    assert torch.equal(got, fp32.to(dtype))
