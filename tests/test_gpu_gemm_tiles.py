"""Layouts and tiles of the GEMM engines at the sizes where a tile, a k block or a vector load ends.

Tolerances: a product of K terms summed in fp32 is within K * 2^-24 of its exact value relative to the sum of magnitudes
(twice that is allowed: the tensor cores do not round every partial sum), and rounding to a 16-bit result adds one
half-ulp of the value: 2^-11 for fp16, 2^-8 for bf16."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    return ops, capi


def _bound(A, W, want, K, half_ulp):
    return half_ulp * np.abs(want) + 2 * K * 2.0 ** -24 * (np.abs(A) @ np.abs(W) + 1) + 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("P,M,N,K,ldb,shared", [
    (1, 128, 64, 64, 64, False), (1, 130, 80, 16, 80, False), (3, 77, 72, 200, 72, True), (2, 300, 8, 24, 16, False),
    (1, 515, 320, 136, 320, False), (2, 2600, 200, 72, 256, True), (8, 1000, 128, 256, 128, True), (1, 129, 512, 513, 512, False)])
def test_weights_in_k_n_layout(dtype, P, M, N, K, ldb, shared):
    """fp16 / bf16 weights as [K, N]: one and several 64-column boxes, part boxes, wide rows, shared and per-branch
    inputs, weight tiles that stay resident (many m tiles) and that ride in the ring."""
    ops, capi = _ops()
    rng = np.random.default_rng(P * 7 + M + N + K)
    lda = (K + 7) // 8 * 8
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)
    A = t(rng.normal(0, 1, ((1 if shared else P), M, lda)))
    W = t(rng.normal(0, 1, (P, K, ldb)) / np.sqrt(K))
    bias = torch.from_numpy(rng.normal(0, 0.3, (P, N)).astype(np.float32)).cuda()
    Y = torch.full((P, M, N), 7.0, dtype=dtype, device="cuda")
    ops.gemm(A, W, Y=Y, bias=bias, batch=P, M=M, N=N, K=K, lda=lda, ldb=ldb, ldy=N,
             strides=(0 if shared else M * lda, K * ldb, N, M * N), bias_kind=capi.XB_BIAS_ROW)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    got, f = Y.double().cpu().numpy(), lambda x: x.double().cpu().numpy()
    for p in range(P):
        a, w = f(A)[0 if shared else p][:, :K], f(W)[p][:, :N]
        want = a @ w + f(bias)[p]
        err = np.abs(got[p] - want)
        assert (err <= _bound(a, w, want, K, 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8)).all(), float(err.max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("epi", ["none", "dice"])
def test_weights_in_k_n_layout_with_fp32_results_keep_the_precision_of_the_cuda_cores(dtype, epi):
    """K fp32 FMAs in order: within K * 2^-24 of the sum of magnitudes in the worst case; the bits of the explicit engine."""
    ops, capi = _ops()
    rng = np.random.default_rng(3)
    M, N, K = 300, 128, 512
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to("cuda", d)
    A, W = t(rng.normal(0, 1, (M, K)), dtype), t(rng.normal(0, 1, (K, N)) / np.sqrt(K), dtype)
    bias = t(rng.normal(0, 0.3, N), torch.float32)
    kw = {} if epi == "none" else dict(epilogue=capi.XB_EPI_DICE, ep=[t(rng.uniform(0.1, 0.5, N), torch.float32) for _ in range(3)])
    got, simt = [ops.gemm(A, W, bias=bias, out_dtype=torch.float32, engine=e, **kw) for e in (capi.XB_GEMM_AUTO, capi.XB_GEMM_SIMT)]
    assert torch.equal(got, simt)
    if epi == "none":
        f = lambda x: x.double().cpu().numpy()
        assert (np.abs(f(got) - (f(A) @ f(W) + f(bias))) <= (K + 2) * 2.0 ** -24 * (np.abs(f(A)) @ np.abs(f(W)) + np.abs(f(bias)))).all()


def test_explicit_tensor_core_engine_still_wants_k_major_weights():
    ops, capi = _ops()
    A, W = torch.zeros((128, 64), dtype=torch.float16, device="cuda"), torch.zeros((64, 64), dtype=torch.float16, device="cuda")
    with pytest.raises(capi.XbError, match="tcgen05 engine needs"):
        ops.gemm(A, W, engine=capi.XB_GEMM_TCGEN05)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("P,M,N,K,dtype", [(1, 1, 1, 1, "f32"), (1, 33, 17, 15, "f32"), (2, 200, 80, 144, "f32"),
                                          (1, 20000, 40, 80, "f32"), (1, 3000, 200, 36, "f32"), (1, 700, 129, 18, "f32"),
                                          (3, 64, 36, 100, "f32"), (2, 130, 45, 37, "f16"), (1, 100, 24, 52, "bf16")])
def test_cuda_core_engine_tiles_and_layouts(ta, tb, P, M, N, K, dtype):
    """Every transpose through both the 16-byte and the element loads (sizes that are and are not multiples of four),
    tiles from 32 x 16 up to 128 x 128, batches."""
    ops, capi = _ops()
    rng = np.random.default_rng(M + N + K + 2 * ta + tb)
    dt = dict(f32=torch.float32, f16=torch.float16, bf16=torch.bfloat16)[dtype]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dt)
    A = t(rng.normal(0, 1, (P, K, M) if ta else (P, M, K)))
    B = t(rng.normal(0, 1, (P, N, K) if tb else (P, K, N)) / np.sqrt(K))
    bias = torch.from_numpy(rng.normal(0, 0.3, (P, M, N)).astype(np.float32)).cuda()
    Y = torch.full((P, M, N), 7.0, dtype=torch.float32, device="cuda")
    ops.gemm(A, B, Y=Y, bias=bias, trans_a=bool(ta), trans_b=bool(tb), alpha=0.5, beta=2.0, batch=P, M=M, N=N, K=K,
             lda=A.shape[2], ldb=B.shape[2], ldy=N, ldbias=N, strides=(M * K, K * N, M * N, M * N),
             bias_kind=capi.XB_BIAS_FULL, engine=capi.XB_GEMM_SIMT)
    f = lambda x: x.double().cpu().numpy()
    for p in range(P):
        a, b = (f(A)[p].T if ta else f(A)[p]), (f(B)[p].T if tb else f(B)[p])
        want = 0.5 * (a @ b) + 2.0 * f(bias)[p]
        err = np.abs(f(Y)[p] - want)
        assert (err <= _bound(a, b, want, K, 2.0 ** -23)).all(), float(err.max())


@pytest.mark.parametrize("P,M,N,K,dtype,out,epi", [
    (1, 128 * 148, 256, 256, "bf16", "bf16", "prelu"),       # whole 256-row tiles, one column of them
    (1, 9500, 512, 320, "f16", "f16", "sigmoid"),            # ragged rows: the second CTA of the last pair has 28 of 128
    (2, 4890, 512, 1000, "f16", "f32", "dice"),              # the last pair's second CTA has no rows; ragged K; batches
    (1, 2432, 2048, 384, "bf16", "f16", "none")])
def test_two_cta_tiles(P, M, N, K, dtype, out, epi):
    ops, capi = _ops()
    rng = np.random.default_rng(M + N + K)
    dt = dict(f16=torch.float16, bf16=torch.bfloat16, f32=torch.float32)
    lda = (K + 7) // 8 * 8
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to("cuda", d)
    A, W = t(rng.normal(0, 1, (P, M, lda)), dt[dtype]), t(rng.normal(0, 1, (P, N, lda)) / np.sqrt(K), dt[dtype])
    W[:, :, K:] = 0
    bias = t(rng.normal(0, 0.3, (P, N)), torch.float32)
    Y = torch.full((P, M, N), 7.0, dtype=dt[out], device="cuda")
    kw = {}
    if epi == "prelu":
        kw = dict(epilogue=capi.XB_EPI_PRELU, ep=(torch.full((1,), 0.25, device="cuda"), None, None), ep_count=1)
    elif epi == "sigmoid":
        kw = dict(epilogue=capi.XB_EPI_SIGMOID)
    elif epi == "dice":
        ep = [t(rng.uniform(0.1, 0.5, (P, N)), torch.float32) for _ in range(3)]
        kw = dict(epilogue=capi.XB_EPI_DICE, ep=ep, stride_ep=N)
    ops.gemm(A, W, Y=Y, bias=bias, trans_b=True, batch=P, M=M, N=N, K=K, lda=lda, ldb=lda, ldy=N,
             strides=(M * lda, N * lda, N, M * N), bias_kind=capi.XB_BIAS_ROW, **kw)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    half_ulp = dict(f16=2.0 ** -11, bf16=2.0 ** -8, f32=2.0 ** -23)[out]
    for p in range(P):
        a, w = A[p, :, :K].double(), W[p, :, :K].double()
        pre = a @ w.t() + bias[p].double()
        want = pre
        if epi == "prelu":
            want = torch.where(pre < 0, pre * 0.25, pre)
        elif epi == "sigmoid":
            want = pre.sigmoid()
        elif epi == "dice":
            g, m, v = [e[p].double() for e in ep]
            s = ((pre - m) / (v + 1e-8).sqrt()).sigmoid()
            want = (1 - s) * g * pre + s * pre
        # the activations' slopes are at most about 1 (sigmoid, PReLU) and 4 (Dice with var >= 0.1); __expf and the fast
        # division add 2^-20 of the value
        scale = a.abs() @ w.abs().t() + 1
        tol = (half_ulp + 2.0 ** -20) * want.abs() + (4 if epi == "dice" else 1) * 2 * K * 2.0 ** -24 * scale
        assert ((Y[p].double() - want).abs() <= tol).all(), float((Y[p].double() - want).abs().max())
