"""Pooling calls at the sizes where the way counts are turned into offsets, or the segments of a warp, change."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _ops():
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    return capi, ops


def _check(batch, groups, max_len, dim, dtype, counts, hashed, seed):
    capi, ops = _ops()
    rng = np.random.default_rng(seed)
    rows = 5000
    w = torch.from_numpy(rng.normal(0, 0.1, (rows, dim)).astype(np.float32)).to(dtype)
    keys = torch.from_numpy((np.arange(rows, dtype=np.int64) + 1) * 7046029254386353) if hashed else None
    table = ops.Table(w.float(), dtype, keys=keys)
    out = torch.full((batch, groups * dim), 9.0, dtype=dtype, device="cuda")
    want = torch.zeros((batch, groups, dim), dtype=torch.float64)
    bound = torch.zeros((batch, groups, dim), dtype=torch.float64)
    gs = []
    for i in range(groups):
        n = rng.integers(0, max_len + 1, batch).astype(np.int32)
        row = rng.integers(0, rows, int(n.sum()))
        vals = rng.uniform(0.5, 1.5, len(row)).astype(np.float32)
        seg = torch.from_numpy(np.repeat(np.arange(batch), n))
        x = w[row].double() * torch.from_numpy(vals).double()[:, None]
        want[:, i].index_add_(0, seg, x)
        bound[:, i].index_add_(0, seg, x.abs())
        ids = torch.from_numpy(row) if keys is None else keys[row]
        segs = torch.from_numpy(n if counts else np.concatenate([[0], np.cumsum(n)]).astype(np.int32))
        gs.append(ops.make_group(table, ids.cuda(), torch.from_numpy(vals).cuda(), segs.cuda(),
                                 [dict(udf=capi.XB_UDF_SUM, out=out, col=i * dim)], dtype, segments_are_offsets=not counts))
    ops.PoolPlan(gs).run()
    err = (out.double().cpu().view(batch, groups, dim) - want).abs()
    # max_len terms summed in fp32, each product rounded once, then the type's half-ulp
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -24
    assert (err <= ulp * want.abs() + (max_len + 1) * 2.0 ** -24 * bound + 1e-7).all(), float(err.max())


@pytest.mark.parametrize("batch", [1, 3, 16, 33, 257, 1023, 1024, 1025])
@pytest.mark.parametrize("dim,dtype,max_len,hashed", [(18, torch.float16, 9, True), (4, torch.float32, 60, False), (64, torch.float32, 3, False)])
def test_counts(batch, dim, dtype, max_len, hashed):
    _check(batch, 2, max_len, dim, dtype, True, hashed, batch)


@pytest.mark.parametrize("batch,groups", [(9500, 4), (30011, 4), (60000, 3)])       # 8, 16 and 32 segments a warp, ragged ends
@pytest.mark.parametrize("dim,dtype", [(32, torch.float16), (64, torch.float16), (8, torch.float32)])
def test_segments_of_a_warp(batch, groups, dim, dtype):
    _check(batch, groups, 8, dim, dtype, False, False, batch + dim)
