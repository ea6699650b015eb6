"""The queue kernel's runs of segments: shorter and longer than its windows of 32, many of them empty or long, groups of unequal
size (the last warps of each have less), every row width, mixed with groups that other kernels take; against index_add in 64
bits. fp32 sums in id order: n roundings of the sum of magnitudes."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,dtype", [(4, torch.float32), (16, torch.float32), (64, torch.float32), (12, torch.float16), (32, torch.float16),
                                       (64, torch.float16), (128, torch.float16)])
@pytest.mark.parametrize("batches", [(39000,), (37900, 5, 70, 1), (15000,) * 20, (300_000, 33)])
@pytest.mark.parametrize("spread", ["even", "gaps", "long"])
def test_runs_of_segments(dim, dtype, batches, spread):
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    rng = np.random.default_rng(dim + len(batches))
    rows = 2000
    table = ops.Table(torch.from_numpy(rng.normal(0, 0.1, (rows, dim)).astype(np.float32)), dtype)
    W = table.buf[:, :dim].double()
    groups, checks = [], []
    for i, B in enumerate(batches):
        n = rng.integers(1, 8, B)
        if spread == "gaps":
            n[rng.random(B) < 0.4] = 0
            n[rng.random(B) < 0.2] += 9
        elif spread == "long":
            n[rng.integers(0, B, max(1, B // 200))] = 300
        if i == 3:
            n[:] = 1                                        # a group for another kernel
        off = torch.from_numpy(np.concatenate([[0], np.cumsum(n)]).astype(np.int32)).cuda()
        ids = torch.from_numpy(rng.integers(-1, rows + 1, int(off[-1]))).cuda()
        out = torch.full((B, dim + 1), 9.0, dtype=dtype, device="cuda")
        udf = capi.XB_UDF_AVG if i % 2 else capi.XB_UDF_SUM
        groups.append(ops.make_group(table, ids, None, off, [dict(udf=udf, out=out)], dtype, segments_are_offsets=True))
        checks.append((off, ids, out, udf))
    ops.PoolPlan(groups).run()
    for off, ids, out, udf in checks:
        lens = off.long().diff()
        known = (ids >= 0) & (ids < rows)
        seg = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), lens)[known]
        want, mag = [torch.zeros((len(lens), dim), dtype=torch.float64, device="cuda").index_add_(0, seg, w[ids[known]]) for w in (W, W.abs())]
        if udf == capi.XB_UDF_AVG:
            want, mag = [x / lens.clamp(min=1)[:, None] for x in (want, mag)]
        eps = 0.0 if dtype == torch.float32 else 2.0 ** -11
        err = (out[:, :dim].double() - want).abs()
        assert (err <= 310 * 2.0 ** -24 * mag + eps * want.abs() + 1e-7).all(), float(err.max())
        assert (out[:, dim] == 9.0).all()


@pytest.mark.parametrize("dim,dtype", [(16, torch.float32), (16, torch.float16), (32, torch.float16), (64, torch.float16)])
@pytest.mark.parametrize("order", ["as drawn", "sorted"])
def test_groups_of_unequal_lists(dim, dtype, order):
    """Shares of a different number of segments for each group, lists sorted by length."""
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    rng = np.random.default_rng(dim)
    rows, spans = 3000, [(1, 9, 20001), (40, 50, 5003), (3, 6, 17), (1, 30, 30_011), (30, 60, 8191)]
    table = ops.Table(torch.from_numpy(rng.normal(0, 0.1, (rows, dim)).astype(np.float32)), dtype)
    W = table.buf[:, :dim].double()
    groups, checks = [], []
    for lo, hi, B in spans:
        n = rng.integers(lo, hi + 1, B)
        n = np.sort(n)[::-1] if order == "sorted" else n
        off = torch.from_numpy(np.concatenate([[0], np.cumsum(n)]).astype(np.int32)).cuda()
        ids = torch.from_numpy(rng.integers(0, rows, int(off[-1]))).cuda()
        out = torch.full((B + 1, dim), 9.0, dtype=dtype, device="cuda")
        groups.append(ops.make_group(table, ids, None, off, [dict(udf=capi.XB_UDF_SUM, out=out)], dtype, segments_are_offsets=True))
        checks.append((off, ids, out))
    ops.PoolPlan(groups).run()
    for off, ids, out in checks:
        seg = torch.repeat_interleave(torch.arange(len(off) - 1, device="cuda"), off.long().diff())
        want, mag = [torch.zeros((len(off) - 1, dim), dtype=torch.float64, device="cuda").index_add_(0, seg, w[ids]) for w in (W, W.abs())]
        eps = 0.0 if dtype == torch.float32 else 2.0 ** -11
        assert ((out[:-1].double() - want).abs() <= 60 * 2.0 ** -24 * mag + eps * want.abs() + 1e-7).all()
        assert (out[-1] == 9.0).all()
