"""The per-step attention engine with the steps of a tile shared by a cluster, and with zero k rows around a list."""
import numpy as np
import pytest
import torch

import orc
import pkg
from test_gpu_attention import _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,n_cand,T,lens", [
    (1, 200, 100, None),            # 2 tiles: clusters of 8, 13 steps a CTA, the last one 9
    (1, 5, 3, None),                # fewer steps than the widest cluster
    (9, 130, 17, None),             # 18 tiles, ragged everywhere
    (2, 128, 100, [0, 3]),          # nothing to walk, and fewer steps than CTAs
    (3, 129, 50, [50, 1, 27]),
    (30, 1000, 20, None)])          # 240 tiles: more than one wave whatever the split
@pytest.mark.parametrize("d,h0,h1,act", [(36, 80, 40, 2), (32, 64, 32, 2), (18, 32, 16, 0)])
@pytest.mark.parametrize("zeros", ["none", "lead", "mixed"])
@pytest.mark.parametrize("scores", [False, True])
def test_steps_shared_by_a_cluster(R, n_cand, T, lens, d, h0, h1, act, zeros, scores):
    if R == 30 and (zeros == "mixed" or d != 36):
        pytest.skip("one shape of the many-tile case is enough")
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    rng = np.random.default_rng(R * 100 + T + d)
    w = _weights(rng, d, h0, h1)
    q = rng.normal(0, 0.5, (R * n_cand, d)).astype(np.float16)
    k = rng.normal(0, 0.5, (R, T, d)).astype(np.float16)
    if zeros != "none":
        for r in range(R):
            k[r, : (r * 7 + T // 2) % (T + 1)] = 0                  # a list right-aligned in its rows, as kAssign leaves it
            if zeros == "mixed":
                k[r, T - 1 - r % T:] = -0.0                         # zero rows at the end, one in the middle
                k[r, T // 2] = 0
    t = torch.from_numpy
    att = ops.DinAttention(t(w["W0"]), t(w["b0"]), t(w["W1"]), t(w["b1"]), t(w["W2"]), float(w["b2"][0]),
                           dice0=[t(w["g0"]), t(w["m0"]), t(w["v0"])], dice1=[t(w["g1"]), t(w["m1"]), t(w["v1"])], act=act)
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda") if lens else None
    sc = torch.zeros((R * n_cand, T), device="cuda") if scores else None
    out = torch.full((R * n_cand, d), 9.0, dtype=torch.float16, device="cuda")
    att(t(q).cuda(), t(k.reshape(R * T, d)).cuda(), R, n_cand, T, out=out, seq_len=sl, scores=sc, engine=capi.XB_GEMM_TCGEN05)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    got = out.float().cpu().numpy()
    for r in {0, 1, R // 2, R - 1} & set(range(R)):
        o, s = orc.din_attention(q[r * n_cand:(r + 1) * n_cand].astype(np.float32), k[r].astype(np.float32), w, act=act,
                                 seq_len=lens[r] if lens else T, use_softmax=False, want_scores=True)
        rows = slice(r * n_cand, (r + 1) * n_cand)
        if scores:
            assert np.abs(sc[rows].cpu().numpy() - s).max() <= 5e-3
        # the bounds of test_gpu_attention.py: fp16 scores against the sum of their magnitudes
        assert (np.abs(got[rows] - o) <= 4e-3 * (1 + np.abs(s) @ np.abs(k[r].astype(np.float32)))).all()


def test_a_request_gets_the_same_bits_alone_and_in_a_batch():
    """One request alone is split over clusters; among enough others it is not. The scores meet in one closing product
    either way."""
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    rng = np.random.default_rng(5)
    R, n_cand, T, d = 80, 256, 100, 36
    w = _weights(rng, d, 80, 40)
    t = torch.from_numpy
    att = ops.DinAttention(t(w["W0"]), t(w["b0"]), t(w["W1"]), t(w["b1"]), t(w["W2"]), float(w["b2"][0]),
                           dice0=[t(w["g0"]), t(w["m0"]), t(w["v0"])], dice1=[t(w["g1"]), t(w["m1"]), t(w["v1"])], act=2)
    q = t(rng.normal(0, 0.5, (R * n_cand, d)).astype(np.float16)).cuda()
    k = rng.normal(0, 0.5, (R, T, d)).astype(np.float16)
    k[3, :61] = 0
    k = t(k.reshape(R * T, d)).cuda()
    all_ = att(q, k, R, n_cand, T, engine=capi.XB_GEMM_TCGEN05)
    for r in (0, 3, 79):
        one = att(q[r * n_cand:(r + 1) * n_cand], k[r * T:(r + 1) * T], 1, n_cand, T, engine=capi.XB_GEMM_TCGEN05)
        assert torch.equal(one, all_[r * n_cand:(r + 1) * n_cand])
    assert ops.device_status() == 0


@pytest.mark.parametrize("R,n_cand,T", [(1, 140, 100), (5, 130, 17), (160, 128, 20)])      # split, split, one wave and more
@pytest.mark.parametrize("lens", [False, True])
def test_scores_that_are_no_finite_numbers_show_through_zero_rows(R, n_cand, T, lens):
    """s * 0 is NaN for such a score: a call that walks every step (because it wants the scores) and one that leaves out
    zero rows agree, whether the odd rows of q meet lists of zeros, short lists or full ones."""
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    rng = np.random.default_rng(R)
    d = 36
    w = _weights(rng, d, 80, 40)
    t = torch.from_numpy
    att = ops.DinAttention(t(w["W0"]), t(w["b0"]), t(w["W1"]), t(w["b1"]), t(w["W2"]), float(w["b2"][0]),
                           dice0=[t(w["g0"]), t(w["m0"]), t(w["v0"])], dice1=[t(w["g1"]), t(w["m1"]), t(w["v1"])], act=2)
    q = rng.normal(0, 0.5, (R, n_cand, d)).astype(np.float16)
    q[:, 3, 5], q[:, 17, 0], q[:, 40, 35] = np.inf, -np.inf, np.nan
    q[:, 60], q[:, 61] = 6e4, -6e4                                     # finite, their scores are not
    k = rng.normal(0, 0.5, (R, T, d)).astype(np.float16)
    for r in range(R):
        kind = r % 5
        if kind == 0:
            k[r] = 0
        elif kind == 1:
            k[r, : T // 2] = 0
        elif kind == 2:
            k[r, T // 3:] = -0.0
        elif kind == 3:
            k[r, : T // 3] = 0
            k[r, T - 2:] = 0
    sl = torch.from_numpy(rng.integers(0, T + 1, R).astype(np.int32)).cuda() if lens else None
    qd, kd = t(q.reshape(R * n_cand, d)).cuda(), t(k.reshape(R * T, d)).cuda()
    call = lambda sc: att(qd, kd, R, n_cand, T, seq_len=sl, scores=sc, engine=capi.XB_GEMM_TCGEN05)
    got, want = call(None).clone(), call(torch.zeros((R * n_cand, T), device="cuda")).clone()
    assert ops.device_status() == 0
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(nan=9.0), want.nan_to_num(nan=9.0))
    rows = got.view(R, n_cand, d)[:, [3, 17, 40]].isfinite().logical_not().all(-1)
    live = sl.cpu() > 0 if lens else torch.ones(R, dtype=torch.bool)
    assert rows[live.cuda()].all() and not rows[~live.cuda()].any()            # an odd q row shows unless its list is empty
