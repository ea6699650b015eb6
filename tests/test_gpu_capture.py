"""The hot path inside a CUDA graph: kernels whose launches overlap the one before give the same bits when replayed."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,requests,n_cand", [("din", 1, 130), ("din", 3, 1000), ("dien", 2, 200)])
def test_forward_replayed_from_a_graph(kind, requests, n_cand):
    pkg.load()
    from x_deeplearning_b200 import dien, din, ops, workloads
    make = workloads.din_model if kind == "din" else workloads.dien_model
    model = make(0, item_rows=5000, cate_rows=500, user_rows=500, emb_sigma=0.5)
    net = (din.DinModel if kind == "din" else dien.DienModel)(model)
    run = (lambda p: net.forward_device(p)) if kind == "din" else (lambda p: net.forward_dien(p)[0])
    reqs = [workloads.din_requests(model, s, requests=requests, n_cand=n_cand) for s in (1, 2)]
    want = []
    for q in reqs:
        want.append(run(net.upload(net.stage(q))).clone())
    p = net.upload(net.stage(reqs[0]))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run(p)
    torch.cuda.current_stream().wait_stream(side)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = run(p)
    for i in (0, 1, 0):
        net.upload(net.stage(reqs[i]))
        for _ in range(3):                         # replays follow one another without a gap
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[i])
    assert ops.device_status() == 0
