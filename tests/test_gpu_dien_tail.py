"""What the DIEN-style model runs around its AUGRU: softmax with an fp16 copy and the fused tower with PReLU, against plain
torch in 64 bits."""
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    return ops, capi, capi.lib()


@pytest.mark.parametrize("n,c", [(1, 16), (33, 20), (500, 64), (131, 65), (77, 100), (40, 101), (9, 128), (35, 129), (64, 256),
                                 (5, 257), (7, 3), (50000, 36)])
def test_softmax_scores(n, c):
    ops, capi, L = _ops()
    g = torch.Generator(device="cuda").manual_seed(n)
    for shift in (0, 1):                                            # rows of whole 16-byte pieces, then misaligned ones
        x = torch.randn(n * c + 1, generator=g, device="cuda")[shift:shift + n * c] * 6
        x[0] = -torch.inf
        y, y16 = torch.full((n, c), 9.0, device="cuda"), torch.full((n, c), 9.0, device="cuda", dtype=torch.float16)
        capi.check(L.xb_softmax_scores(ops.ptr(x), ops.ptr(y), ops.ptr(y16), n, c, ops.stream()))
        want = x.double().view(n, c).softmax(1)
        # __expf of a difference r below zero: 2 + 1.173 r units in the last place, r / 2 more for the rounding of r; the sum of
        # such terms and the division: a few more
        low = x[torch.isfinite(x)].min()
        r = float(x.max() - low)
        assert ((y.double() - want).abs() <= (10 + 1.7 * r) * 2.0 ** -23 * want + 1e-37).all()
        assert torch.equal(y16, y.half())
        z = torch.full_like(y, 9.0)
        capi.check(L.xb_softmax(ops.ptr(x), ops.ptr(z), n, c, 1, capi.XB_F32, ops.stream()))
        assert torch.equal(y, z)
        capi.check(L.xb_softmax(ops.ptr(x), ops.ptr(x), n, c, 1, capi.XB_F32, ops.stream()))       # in place
        assert torch.equal(y.view(-1), x)


@pytest.mark.parametrize("R,n_cand,T,d,du,dims", [(1, 5, 3, 36, 144, (200, 80, 2)), (3, 130, 20, 36, 144, (200, 80, 2)),
                                                  (2, 300, 7, 32, 40, (64, 32, 1)), (150, 129, 2, 16, 8, (48, 24, 8)),
                                                  (160, 200, 2, 36, 30, (77, 33, 3))])
@pytest.mark.parametrize("softmax", [True, False])
def test_tower_with_prelu(R, n_cand, T, d, du, dims, softmax):
    ops, capi, _ = _ops()
    g = torch.Generator().manual_seed(R + d)
    r = lambda *s: torch.randn(s, generator=g)
    n1, n2, n3 = dims
    h = lambda x: x.half().float()
    W1, W2, W3 = h(r(du + 5 * d, n1) / (du + 5 * d) ** 0.5), h(r(n1, n2) / n1 ** 0.5), h(r(n2, n3) / n2 ** 0.5)
    b1, b2, b3 = r(n1) * 0.1, r(n2) * 0.1, r(n3) * 0.1
    s1, s2 = torch.rand(n1, generator=g) * 0.5, torch.rand(n2, generator=g) * 0.5
    user, q, k, att = [h(r(*s)).half().cuda() for s in ((R, du), (R * n_cand, d), (R * T, d), (R * n_cand, d))]
    tower = ops.DinTower(d, du, W1, b1, [s1], W2, b2, [s2], W3, b3, softmax=softmax, act=capi.XB_ACT_PRELU)
    got = tower(user, q, k, att, R, n_cand, T).double().cpu()
    D = lambda x: x.double().cpu()
    his = D(k).view(R, T, d).sum(1).half().double().repeat_interleave(n_cand, 0)
    x = torch.cat([D(user).repeat_interleave(n_cand, 0), D(q), his, (D(q) * his).half().double(), D(att), (D(q) - his).half().double()], 1)
    for W, b, s in ((W1, b1, s1), (W2, b2, s2)):
        x = x @ W.double() + b.double()
        x = torch.where(x < 0, x * s.double(), x).half().double()
    want = x @ W3.double() + b3.double()
    # two roundings to fp16 (2^-11 of the value) carried through the layers after them; his_sum may round to its neighbour
    tol = 2.0 ** -9 * (1 + want.abs().max()) * 1.5
    if softmax:
        want = want.softmax(1)
    assert (got - want).abs().max() <= tol, (float((got - want).abs().max()), float(tol))


@pytest.mark.parametrize("R,n_cand,T,d,du,dims", [(150, 129, 3, 36, 144, (200, 80, 2)), (310, 100, 2, 20, 8, (48, 24, 5))])
def test_dice_tower_over_several_tiles_a_block(R, n_cand, T, d, du, dims):
    """More tiles than SMs: a block begins its next tile between the two epilogues of the one before."""
    ops, capi, _ = _ops()
    g = torch.Generator().manual_seed(R)
    r = lambda *s: torch.randn(s, generator=g)
    u = lambda n, lo, hi: torch.rand(n, generator=g) * (hi - lo) + lo
    n1, n2, n3 = dims
    h = lambda x: x.half().float()
    W1, W2, W3 = h(r(du + 5 * d, n1) / (du + 5 * d) ** 0.5), h(r(n1, n2) / n1 ** 0.5), h(r(n2, n3) / n2 ** 0.5)
    b1, b2, b3 = r(n1) * 0.1, r(n2) * 0.1, r(n3) * 0.1
    dice = [[u(n, 0, 0.5), u(n, -0.1, 0.1), u(n, 0.5, 1.5)] for n in (n1, n2)]
    user, q, k, att = [h(r(*s)).half().cuda() for s in ((R, du), (R * n_cand, d), (R * T, d), (R * n_cand, d))]
    got = ops.DinTower(d, du, W1, b1, dice[0], W2, b2, dice[1], W3, b3, softmax=False)(user, q, k, att, R, n_cand, T).double().cpu()
    D = lambda x: x.double().cpu()
    his = D(k).view(R, T, d).sum(1).half().double().repeat_interleave(n_cand, 0)
    x = torch.cat([D(user).repeat_interleave(n_cand, 0), D(q), his, (D(q) * his).half().double(), D(att), (D(q) - his).half().double()], 1)
    for W, b, (ga, mu, va) in ((W1, b1, dice[0]), (W2, b2, dice[1])):
        x = x @ W.double() + b.double()
        p = ((x - mu.double()) / (va.double() + 1e-8).sqrt()).sigmoid()
        x = (1 - p) * ga.double() * x + p * x
    want = x @ W3.double() + b3.double()
    # Dice on fp16 pairs: half-precision tanh (5e-4) and three roundings (2^-11) of a value, twice, and the logits' rounding
    tol = 4e-3 * (1 + float((x.abs() @ W3.double().abs()).max()))
    assert (got - want).abs().max() <= tol, (float((got - want).abs().max()), tol)


@pytest.mark.parametrize("R,n_cand,T,d,du,dims", [(16, 500, 100, 36, 144, (200, 80, 2)), (3, 130, 20, 32, 128, (64, 32, 2)), (40, 64, 50, 16, 8, (48, 24, 8))])
def test_prelu_tower_rounds_where_its_layers_do(R, n_cand, T, d, du, dims):
    """The fused tower and the chain that it stands for (input kernel, three GEMMs): the same fp16 layer input and activations, so
    they differ by the order of fp32 sums and by the few activations that this moves to the next fp16 number. A further rounding of
    a layer's input (his_sum before its products, for one) moves them by 2^-13 of the layer's spread and more."""
    ops, capi, L = _ops()
    g = torch.Generator(device="cuda").manual_seed(R + d)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    n1, n2, n3 = dims
    W1, W2, W3 = r(du + 5 * d, n1) / (du + 5 * d) ** 0.5, r(n1, n2) / n1 ** 0.5, r(n2, n3) / n2 ** 0.5
    b1, b2, b3 = r(n1) * 0.1, r(n2) * 0.1, r(n3) * 0.1
    s1, s2 = torch.rand(n1, generator=g, device="cuda") * 0.5, torch.rand(n2, generator=g, device="cuda") * 0.5
    user, q, k, att = [r(*s).half() for s in ((R, du), (R * n_cand, d), (R * T, d), (R * n_cand, d))]
    c = lambda t: t.cpu()
    tower = ops.DinTower(d, du, c(W1), c(b1), [c(s1)], c(W2), c(b2), [c(s2)], c(W3), c(b3), softmax=False, act=capi.XB_ACT_PRELU)
    got = tower(user, q, k, att, R, n_cand, T)
    N, ldx = R * n_cand, (du + 5 * d + 7) // 8 * 8
    X = torch.empty((N, ldx), dtype=torch.float16, device="cuda")
    capi.check(L.xb_din_tower_input(ops.ptr(user), du, ops.ptr(q), d, ops.ptr(k), d, ops.ptr(att), d, ops.ptr(X), ldx, R, n_cand, T, d, du,
                                    ops.stream()))
    prelu = lambda s: dict(epilogue=capi.XB_EPI_PRELU, ep=(s, None, None), ep_count=s.numel())
    y = ops.gemm(X, ops.pack_weight_kmajor(W1, ldk=ldx), bias=b1, trans_b=True, M=N, N=n1, K=ldx, **prelu(s1))
    y = ops.gemm(y, ops.pack_weight_kmajor(W2), bias=b2, trans_b=True, M=N, N=n2, K=n1, **prelu(s2))
    want = ops.gemm(y, ops.pack_weight_kmajor(W3), bias=b3, trans_b=True, M=N, N=n3, K=n2, out_dtype=torch.float32)
    # one activation in some thirty meets another fp16 neighbour (fp32 sums of a few hundred terms, 2^-21 apart, against steps of
    # 2^-10): 2^-10 / 30^0.5 of a value at the most, where every rounding moved would be 2^-11 / 3^0.5 = 2.8e-4
    assert float((got - want).double().norm() / want.double().norm()) < 8e-5


@pytest.mark.parametrize("n,c", [(2000, 100), (9000, 37), (5000, 255), (2047, 64), (3000, 132)])
def test_softmax_of_fp16_rows_computes_as_that_of_fp32_ones(n, c):
    """A warp a row for either type where the eight lanes a row of many aligned fp32 rows are not faster: the same sums."""
    ops, capi, L = _ops()
    x = (torch.randn((n, c), generator=torch.Generator(device="cuda").manual_seed(c), device="cuda") * 3).half()
    y16, y32 = torch.empty_like(x), torch.empty((n, c), device="cuda")
    capi.check(L.xb_softmax(ops.ptr(x), ops.ptr(y16), n, c, 1, capi.XB_F16, ops.stream()))
    capi.check(L.xb_softmax(ops.ptr(x.float()), ops.ptr(y32), n, c, 1, capi.XB_F32, ops.stream()))
    assert torch.equal(y16, y32.half())
