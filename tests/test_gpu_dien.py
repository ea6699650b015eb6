"""DIEN-style model (GRU -> attention scores -> AUGRU -> PReLU tower): GPU pipeline against the op-by-op CPU
oracle. The AUGRU cell has no counterpart in the reference's inference code, so this parity is against the
restated training-side cell only."""
import numpy as np
import pytest
import torch

import dien_oracle
import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("augru_engine", [1, 0])        # CUDA-core AUGRU, then the tcgen05 one (XB_GEMM_AUTO picks it)
@pytest.mark.parametrize("R,n_cand,emb_sigma", [(2, 64, 0.5), (1, 1000, 0.3)])
def test_dien_probabilities_match_oracle(R, n_cand, emb_sigma, augru_engine):
    pkg.load()
    from x_deeplearning_b200 import dien, ops, workloads
    model = workloads.dien_model(0, item_rows=20000, cate_rows=500, user_rows=3000, emb_sigma=emb_sigma)
    req = workloads.din_requests(model, 5, requests=R, n_cand=n_cand)
    want, wparts = dien_oracle.forward(model, req)
    net = dien.DienModel(model, augru_engine=augru_engine)
    p = net.upload(net.stage(req))
    prob, parts = net.forward_dien(p)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    f = lambda t: t.float().cpu().numpy()
    T, H = 100, 36
    np.testing.assert_allclose(f(parts["hseq"]).reshape(R, T, H), wparts["hseq"], rtol=0, atol=4e-3)      # fp16 GRU states
    np.testing.assert_allclose(f(parts["scores"]), wparts["scores"], rtol=0, atol=2e-3)                 # softmax over steps
    np.testing.assert_allclose(f(parts["final"]), wparts["final"], rtol=0, atol=8e-3)                   # fp16 AUGRU state
    got = f(prob)
    assert np.abs(got - want).max() <= 4e-3, np.abs(got - want).max()
    assert np.abs(got.sum(1) - 1).max() < 1e-5


@pytest.mark.parametrize("tower", [(300, 80, 2), (200, 150, 2)])
def test_towers_beyond_the_fused_kernel(tower):
    """Layers wider than the fused tower takes run as GEMMs."""
    pkg.load()
    from x_deeplearning_b200 import dien, workloads
    model = workloads.dien_model(0, item_rows=2000, cate_rows=100, user_rows=30, emb_sigma=0.3)
    rng, t = np.random.default_rng(1), model["dien_tower"]
    w = lambda k, n: rng.normal(0, 1 / np.sqrt(k), (k, n)).astype(np.float16).astype(np.float32)
    t["W1"], t["W2"], t["W3"] = w(t["W1"].shape[0], tower[0]), w(tower[0], tower[1]), w(tower[1], tower[2])
    for i, n in enumerate(tower):
        t["b%d" % (i + 1)] = np.zeros(n, np.float32)
    t["slope1"], t["slope2"] = np.full(tower[0], 0.25, np.float32), np.full(tower[1], 0.25, np.float32)
    model["dims"]["tower"] = tower
    req = workloads.din_requests(model, 5, requests=2, n_cand=40)
    net = dien.DienModel(model)
    p = net.upload(net.stage(req))
    got = net.forward_dien(p)[0].cpu().numpy()
    want = dien_oracle.forward(model, req)[0]
    assert np.abs(got - want).max() <= 4e-3, np.abs(got - want).max()
