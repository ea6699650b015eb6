"""GRU and tensor-core AUGRU at the sizes where a chunk of steps, a lane quarter or a column group ends, against the
oracle. Tolerances are those of test_gpu_rnn.py: fp32 rounding over the recurrence for the GRU, fp16 operands and gates
for the tensor-core AUGRU."""
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


@pytest.mark.parametrize("B,T,H", [(2, 1, 16), (3, 64, 17), (2, 65, 32), (5, 129, 33), (1, 63, 48), (2, 200, 49), (2, 70, 64)])
def test_gru_chunks_and_widths(B, T, H):
    ops, capi, L = _ops()
    rng = np.random.default_rng(B + T + H)
    r = lambda a: torch.from_numpy(a.astype(np.float32)).cuda()
    x = rng.normal(0, 1, (B, T, H))
    x[0, : T // 2 + 1 if T > 1 else 0] = 0             # the list begins in the middle, for long ones in a later chunk
    Wi, Wh = rng.normal(0, 1 / np.sqrt(H), (H, 3 * H)), rng.normal(0, 1 / np.sqrt(H), (H, 3 * H))
    bi, bh = rng.normal(0, 0.1, 3 * H), rng.normal(0, 0.1, 3 * H)
    dx, dWi, dWh, dbi, dbh = r(x), r(Wi), r(Wh), r(bi), r(bh)
    f = lambda t: t.float().cpu().numpy()
    want = orc.gru(f(dx), f(dWh), f(dWi), f(dbh), f(dbi))
    for y in (torch.full_like(dx, 9.0), dx):             # into another tensor, then in place
        capi.check(L.xb_gru(ops.ptr(dx), ops.ptr(y), B, T, H, ops.ptr(dWi), ops.ptr(dWh), ops.ptr(dbi), ops.ptr(dbh),
                            capi.XB_F32, ops.stream()))
        np.testing.assert_allclose(f(y), want, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("H", [4, 10, 12, 18, 20, 26, 28, 34, 36, 42, 44, 50, 52, 58, 60])
@pytest.mark.parametrize("R,n_cand,T", [(2, 129, 6)])
def test_augru_column_groups(H, R, n_cand, T):
    ops, capi, L = _ops()
    rng = np.random.default_rng(H)
    h16 = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", torch.float16)
    x, att = rng.normal(0, 0.7, (R, T, H)), rng.dirichlet(np.ones(T) * 0.3, R * n_cand)
    Wg, bg = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, 2 * H)), rng.normal(0.5, 0.2, 2 * H)
    Wc, bc = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, H)), rng.normal(0, 0.1, H)
    dx, da, dWg, dbg, dWc, dbc = h16(x), h16(att), h16(Wg), h16(bg), h16(Wc), h16(bc)
    y = torch.full((R * n_cand, H), 9.0, dtype=torch.float16, device="cuda")
    capi.check(L.xb_augru_shared(ops.ptr(dx), ops.ptr(da), ops.ptr(y), R, n_cand, T, H, ops.ptr(dWg), ops.ptr(dbg),
                                 ops.ptr(dWc), ops.ptr(dbc), capi.XB_GEMM_TCGEN05, ops.stream()))
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    f = lambda t: t.float().cpu().numpy()
    want = orc.augru(np.repeat(f(dx), n_cand, axis=0), f(da), f(dWg), f(dbg), f(dWc), f(dbc))[:, T - 1, :]
    np.testing.assert_allclose(f(y), want, rtol=0, atol=8e-3)


@pytest.mark.parametrize("H", [1, 5, 16, 32, 33, 64])
@pytest.mark.parametrize("R,n_cand,T", [(2, 7, 33), (1, 4, 64), (3, 1, 1)])
def test_augru_shared_in_fp32(H, R, n_cand, T):
    """Widths without selector slots take the fp32 kernel: chunks of 32 steps, four candidates a block."""
    ops, capi, L = _ops()
    rng = np.random.default_rng(H + T)
    h16 = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", torch.float16)
    x, att = rng.normal(0, 0.7, (R, T, H)), rng.dirichlet(np.ones(T) * 0.3, R * n_cand)
    Wg, bg = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, 2 * H)), rng.normal(0.5, 0.2, 2 * H)
    Wc, bc = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, H)), rng.normal(0, 0.1, H)
    dx, da, dWg, dbg, dWc, dbc = h16(x), h16(att), h16(Wg), h16(bg), h16(Wc), h16(bc)
    y = torch.full((R * n_cand, H), 9.0, dtype=torch.float16, device="cuda")
    capi.check(L.xb_augru_shared(ops.ptr(dx), ops.ptr(da), ops.ptr(y), R, n_cand, T, H, ops.ptr(dWg), ops.ptr(dbg),
                                 ops.ptr(dWc), ops.ptr(dbc), capi.XB_GEMM_SIMT, ops.stream()))
    f = lambda t: t.float().cpu().numpy()
    want = orc.augru(np.repeat(f(dx), n_cand, axis=0), f(da), f(dWg), f(dbg), f(dWc), f(dbc))[:, T - 1, :]
    # fp32 throughout (2e-5 over the recurrence, as for the GRU), then one fp16 rounding: half an ulp of values below 1
    np.testing.assert_allclose(f(y), want, rtol=0, atol=2.0 ** -12 + 2e-5)
