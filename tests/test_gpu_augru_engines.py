"""The two tensor-core engines behind xb_augru_shared (few tiles: warp-level MMAs, many: tcgen05) over lists longer than a chunk
of 128 steps, ragged tiles of four and of eight warps, and a candidate whose scores are no numbers, which no other candidate
may see. Tolerance as in test_gpu_rnn.py."""
import numpy as np
import pytest
import torch

import orc
import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,T", [(36, 127), (36, 128), (36, 129), (36, 200), (4, 257), (60, 130), (18, 5)])
@pytest.mark.parametrize("R,n_cand", [(1, 17), (2, 65), (16, 1000), (80, 130)])
def test_augru_over_chunks_of_steps(H, T, R, n_cand):
    pkg.load()
    from x_deeplearning_b200 import ops, capi
    rng = np.random.default_rng(H + T)
    h16 = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", torch.float16)
    x, att = rng.normal(0, 0.7, (R, T, H)), rng.dirichlet(np.ones(T) * 0.3, R * n_cand)
    Wg, bg = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, 2 * H)), rng.normal(0.5, 0.2, 2 * H)
    Wc, bc = rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, H)), rng.normal(0, 0.1, H)
    dx, da, dWg, dbg, dWc, dbc = h16(x), h16(att), h16(Wg), h16(bg), h16(Wc), h16(bc)
    bad = n_cand // 2
    da[bad] = torch.nan
    y = torch.full((R * n_cand + 1, H), 9.0, dtype=torch.float16, device="cuda")
    capi.check(capi.lib().xb_augru_shared(ops.ptr(dx), ops.ptr(da), ops.ptr(y), R, n_cand, T, H, ops.ptr(dWg), ops.ptr(dbg),
                                          ops.ptr(dWc), ops.ptr(dbc), capi.XB_GEMM_TCGEN05, ops.stream()))
    assert (y[-1] == 9.0).all() and y[bad].isnan().all()
    few = [i for r in {0, R - 1} for i in range(r * n_cand, (r + 1) * n_cand) if i != bad][:200] + [R * n_cand - 1]
    f = lambda t: t.float().cpu().numpy()
    want = orc.augru(f(dx)[np.array(few) // n_cand], f(da)[few], f(dWg), f(dbg), f(dWc), f(dbc))[:, T - 1, :]
    np.testing.assert_allclose(f(y)[few], want, rtol=0, atol=8e-3)


def _augru(R, n_cand, T, H, seed):
    from x_deeplearning_b200 import ops, capi
    rng = np.random.default_rng(seed)
    h16 = lambda a: torch.from_numpy(a.astype(np.float32)).to("cuda", torch.float16)
    x, att = h16(rng.normal(0, 0.7, (R, T, H))), h16(rng.dirichlet(np.ones(T) * 0.3, R * n_cand))
    w = [h16(rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, 2 * H))), h16(rng.normal(0.5, 0.2, 2 * H)),
         h16(rng.normal(0, 1 / np.sqrt(2 * H), (2 * H, H))), h16(rng.normal(0, 0.1, H))]

    def run(requests, engine):
        y = torch.empty((requests * n_cand, H), dtype=torch.float16, device="cuda")
        capi.check(capi.lib().xb_augru_shared(ops.ptr(x), ops.ptr(att), ops.ptr(y), requests, n_cand, T, H, *[ops.ptr(t) for t in w],
                                              engine, ops.stream()))
        return y
    return x, att, w, run


@pytest.mark.parametrize("H,T", [(36, 100), (4, 257), (60, 130)])
@pytest.mark.parametrize("n_cand", [17, 200])
def test_the_named_engine_whatever_the_number_of_tiles(H, T, n_cand):
    """A candidate's state does not depend on the call's size where the engine is named: few tiles and more than any GPU has SMs."""
    pkg.load()
    from x_deeplearning_b200 import capi
    run = _augru(300, n_cand, T, H, 1)[3]
    many = run(300, capi.XB_GEMM_TCGEN05)
    for few in (1, 3):
        assert torch.equal(run(few, capi.XB_GEMM_TCGEN05), many[:few * n_cand])


@pytest.mark.parametrize("H,T", [(36, 127), (36, 128), (36, 129), (36, 200), (4, 257), (60, 130), (18, 5)])
@pytest.mark.parametrize("R,n_cand", [(1, 17), (2, 65), (16, 1000)])
def test_few_tiles_by_the_engine_that_the_library_picks(H, T, R, n_cand):
    pkg.load()
    from x_deeplearning_b200 import capi
    x, att, w, run = _augru(R, n_cand, T, H, H + T)
    bad = n_cand // 2
    att[bad] = torch.nan
    y = run(R, capi.XB_GEMM_AUTO)
    assert y[bad].isnan().all()
    few = [i for r in {0, R - 1} for i in range(r * n_cand, (r + 1) * n_cand) if i != bad][:200] + [R * n_cand - 1]
    f = lambda t: t.float().cpu().numpy()
    want = orc.augru(f(x)[np.array(few) // n_cand], f(att)[few], *[f(t) for t in w])[:, T - 1, :]
    np.testing.assert_allclose(f(y)[few], want, rtol=0, atol=8e-3)


@pytest.mark.parametrize("H", [4, 18, 36, 60])
@pytest.mark.parametrize("R,n_cand", [(1, 40), (3, 300)])
def test_both_engines_round_in_the_same_places(H, R, n_cand):
    """One input column and one state column a gate, that with weight 1: every sum has one product of each, and what is left of it
    after its roundings to fp16 is exact in fp32 (states are multiples of 2^-24, sums below 1 where a state is small)."""
    pkg.load()
    from x_deeplearning_b200 import capi
    x, att, w, run = _augru(R, n_cand, 30, H, H + R)
    rng = np.random.default_rng(H)
    values = lambda *s: torch.from_numpy(rng.uniform(0.5, 0.7, s) * rng.choice([-1, 1], s)).to("cuda", torch.float16)
    x.zero_()
    x[:, :, 1] = values(R, 30)
    for W in w:
        W.zero_()
    w[0][1], w[2][1] = values(2 * H), values(H)
    eye = torch.eye(H, device="cuda", dtype=torch.float16)
    w[0][H:, :H], w[0][H:, H:], w[2][H:] = eye, eye, eye
    assert torch.equal(run(R, capi.XB_GEMM_AUTO), run(R, capi.XB_GEMM_TCGEN05))


@pytest.mark.parametrize("H", [4, 10, 12, 18, 20, 26, 28, 34, 36, 42, 44, 50, 52, 58, 60])
@pytest.mark.parametrize("R,n_cand,T", [(1, 40, 100), (5, 1000, 100), (2, 65, 131)])
def test_both_engines_give_the_same_states(H, R, n_cand, T):
    """The same chunks in k, the terms of x_t among them, and the same roundings: equal bits, whichever the call's size picks."""
    pkg.load()
    from x_deeplearning_b200 import capi
    run = _augru(R, n_cand, T, H, H + R)[3]
    assert torch.equal(run(R, capi.XB_GEMM_AUTO), run(R, capi.XB_GEMM_TCGEN05))
