"""GRU / AUGRU kernels against the CPU oracle (GRU pinned by the reference fixtures, AUGRU unpinned)."""
import numpy as np
import pytest
import torch

import orc
import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    return ops, capi, capi.lib()


@pytest.mark.parametrize("B,T,H,dtype,tol", [(1000, 100, 36, torch.float32, 2e-5), (7, 5, 64, torch.float32, 2e-5),
                                              (33, 20, 36, torch.float16, 4e-3), (3, 1, 1, torch.float32, 1e-6)])
def test_gru_matches_oracle(B, T, H, dtype, tol):
    ops, capi, L = _ops()
    rng = np.random.default_rng(B + T + H)
    r = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", dtype)
    x = rng.normal(0, 1, (B, T, H))
    x[: B // 3, : T // 2] = 0                      # leading padding steps
    Wi, Wh = rng.normal(0, 1 / np.sqrt(H), (H, 3 * H)), rng.normal(0, 1 / np.sqrt(H), (H, 3 * H))
    bi, bh = rng.normal(0, 0.1, 3 * H), rng.normal(0, 0.1, 3 * H)
    dx, dWi, dWh, dbi, dbh = r(x), r(Wi), r(Wh), r(bi), r(bh)
    y = torch.empty_like(dx)
    capi.check(L.xb_gru(ops.ptr(dx), ops.ptr(y), B, T, H, ops.ptr(dWi), ops.ptr(dWh), ops.ptr(dbi), ops.ptr(dbh),
                        ops.dt(dx), ops.stream()))
    f = lambda t: t.float().cpu().numpy()
    want = orc.gru(f(dx), f(dWh), f(dWi), f(dbh), f(dbi))
    np.testing.assert_allclose(f(y), want, rtol=tol, atol=tol)
    if B >= 3 and T >= 2:
        assert (f(y)[0, : T // 2] == 0).all()


@pytest.mark.parametrize("B,T,H,dtype,tol", [(1000, 100, 36, torch.float32, 2e-5), (5, 9, 16, torch.float16, 4e-3)])
def test_augru_matches_oracle(B, T, H, dtype, tol):
    ops, capi, L = _ops()
    rng = np.random.default_rng(B + H)
    r = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", dtype)
    x, att = rng.normal(0, 1, (B, T, H)), rng.uniform(0, 1, (B, T))
    Wg, bg = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, 2 * H)), rng.normal(0, 0.1, 2 * H)
    Wc, bc = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, H)), rng.normal(0, 0.1, H)
    dx, da, dWg, dbg, dWc, dbc = r(x), r(att), r(Wg), r(bg), r(Wc), r(bc)
    y = torch.empty_like(dx)
    capi.check(L.xb_augru(ops.ptr(dx), ops.ptr(da), ops.ptr(y), B, T, H, ops.ptr(dWg), ops.ptr(dbg), ops.ptr(dWc),
                          ops.ptr(dbc), ops.dt(dx), ops.stream()))
    f = lambda t: t.float().cpu().numpy()
    want = orc.augru(f(dx), f(da), f(dWg), f(dbg), f(dWc), f(dbc))
    np.testing.assert_allclose(f(y), want, rtol=tol, atol=tol)


@pytest.mark.parametrize("engine", ["simt", "tc"])
@pytest.mark.parametrize("R,n_cand,T,H", [(2, 300, 100, 36), (3, 130, 7, 36), (1, 5, 1, 20)])
def test_augru_over_a_shared_sequence_matches_oracle(engine, R, n_cand, T, H):
    """xb_augru_shared: every candidate of a request walks the request's sequence with its own scores; only the final
    state is kept. The tcgen05 engine keeps the state in fp32 and rounds it to fp16 as an MMA operand each step."""
    ops, capi, L = _ops()
    rng = np.random.default_rng(R * 1000 + n_cand + T)
    h16 = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", torch.float16)
    x, att = rng.normal(0, 0.7, (R, T, H)), rng.dirichlet(np.ones(T) * 0.3, R * n_cand)      # softmax-like scores
    Wg, bg = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, 2 * H)), rng.normal(0.5, 0.2, 2 * H)
    Wc, bc = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, H)), rng.normal(0, 0.1, H)
    dx, da, dWg, dbg, dWc, dbc = h16(x), h16(att), h16(Wg), h16(bg), h16(Wc), h16(bc)
    y = torch.full((R * n_cand, H), 9.0, dtype=torch.float16, device="cuda")
    eng = capi.XB_GEMM_SIMT if engine == "simt" else capi.XB_GEMM_TCGEN05
    capi.check(L.xb_augru_shared(ops.ptr(dx), ops.ptr(da), ops.ptr(y), R, n_cand, T, H, ops.ptr(dWg), ops.ptr(dbg),
                                 ops.ptr(dWc), ops.ptr(dbc), eng, ops.stream()))
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    f = lambda t: t.float().cpu().numpy()
    xs = np.repeat(f(dx), n_cand, axis=0)                                       # [R * n_cand, T, H]
    want = orc.augru(xs, f(da), f(dWg), f(dbg), f(dWc), f(dbc))[:, T - 1, :]
    tol = 4e-3 if engine == "simt" else 8e-3
    np.testing.assert_allclose(f(y), want, rtol=0, atol=tol)


def test_augru_tcgen05_engine_declines_shapes_without_selector_slots():
    ops, capi, L = _ops()
    z = torch.zeros(64 * 64 * 4, dtype=torch.float16, device="cuda")
    rc = L.xb_augru_shared(ops.ptr(z), ops.ptr(z), ops.ptr(z), 1, 4, 3, 32, ops.ptr(z), ops.ptr(z), ops.ptr(z), ops.ptr(z),
                           capi.XB_GEMM_TCGEN05, ops.stream())
    assert rc == -2 and b"tcgen05 engine" in L.xb_last_error()


@pytest.mark.parametrize("B,T,H", [(8, 100, 36), (5, 70, 64), (40, 33, 16), (3, 129, 20)])
def test_gru_of_fp16_sequences_computes_as_that_of_fp32_ones(B, T, H):
    """The data type is that of the arrays: the state, the sums and the gates are the same fp32 numbers, so the fp16 result is the
    rounding of the fp32 one over the same inputs."""
    ops, capi, L = _ops()
    g = torch.Generator(device="cuda").manual_seed(B + T + H)
    h16 = lambda sd, *s: (torch.randn(s, generator=g, device="cuda") * sd).half()
    a = [h16(1, B, T, H), h16(H ** -0.5, H, 3 * H), h16(H ** -0.5, H, 3 * H), h16(0.1, 3 * H), h16(0.1, 3 * H)]
    got = []
    for t in (a, [v.float() for v in a]):
        y = torch.empty_like(t[0])
        capi.check(L.xb_gru(ops.ptr(t[0]), ops.ptr(y), B, T, H, *[ops.ptr(v) for v in t[1:]], ops.dt(y), ops.stream()))
        got.append(y)
    assert torch.equal(got[0], got[1].half())


def test_gru_adds_its_recurrent_sums_by_quarters_of_the_units():
    """Units 0 and 16 have the same state and weights 2^30 and -2^30: in the quarter that both belong to they cancel before the term
    of unit 4, which belongs to another, is added. Added between the two it would be lost."""
    ops, capi, L = _ops()
    B, H = 3, 20
    g = torch.Generator().manual_seed(7)
    r = lambda *s: torch.randn(s, generator=g)
    x, Wi, Wh, bi = r(B, 2, H), r(H, 3 * H) / H ** 0.5, torch.zeros((H, 3 * H)), r(3 * H) * 0.1
    for k in range(3):
        Wi[:, k * H + 16], bi[k * H + 16] = Wi[:, k * H], bi[k * H]
    Wh[0, 2 * H:], Wh[4, 2 * H:], Wh[16, 2 * H:] = 2.0 ** 30, 1.0, -2.0 ** 30
    dx, dWi, dWh, dbi, dbh = x.cuda(), Wi.cuda(), Wh.cuda(), bi.cuda(), torch.zeros(3 * H).cuda()
    y = torch.empty_like(dx)
    capi.check(L.xb_gru(ops.ptr(dx), ops.ptr(y), B, 2, H, ops.ptr(dWi), ops.ptr(dWh), ops.ptr(dbi), ops.ptr(dbh), capi.XB_F32, ops.stream()))
    h = torch.zeros((B, H), dtype=torch.float64)
    for t in range(2):
        pre, rec = x[:, t].double() @ Wi.double() + bi.double(), h[:, 4:5]
        reset, z = pre[:, :H].sigmoid(), pre[:, H:2 * H].sigmoid()
        c = (pre[:, 2 * H:] + reset * rec).tanh()
        h = c + z * (h - c)
        assert (y[:, t].double().cpu() - h).abs().max() <= 2e-5


@pytest.mark.parametrize("H", [22, 32, 36, 42, 43, 48, 64])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_gru_of_many_sequences(H, dtype):
    """More sequences than are resident at a time, under another register bound: each has the bits that it has in a small call."""
    ops, capi, L = _ops()
    B, T = 5 * torch.cuda.get_device_properties(0).multi_processor_count + 3, 70
    g = torch.Generator(device="cuda").manual_seed(H)
    r = lambda sd, *s: (torch.randn(s, generator=g, device="cuda") * sd).to(dtype)
    x, w = r(1, B, T, H), [r(H ** -0.5, H, 3 * H), r(H ** -0.5, H, 3 * H), r(0.1, 3 * H), r(0.1, 3 * H)]
    x[::7, :T // 2] = 0

    def run(x):
        y = torch.empty_like(x)
        capi.check(L.xb_gru(ops.ptr(x), ops.ptr(y), len(x), T, H, *[ops.ptr(v) for v in w], ops.dt(y), ops.stream()))
        return y
    many = run(x)
    for i in range(0, B, 100):
        assert torch.equal(run(x[i:i + 100]), many[i:i + 100])
