"""The sharded step of one rank in one call, which pools the caller's lists in place, against the same step in stages, which
routes them through buckets: the same bits for every kernel the pooling may take (short lists, long ones, few and many of
them, rows wider than the fast kernels' limit), tables whose segments do not end with a feature group, odd output strides, ids
no table has, offsets that end before the ids do, and no ids at all."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _both(table_segments, groups, mean, dim, table_dtype, partial, out_dtype, pad, tail, seed):
    from x_deeplearning_b200 import ops, sharded
    rng = np.random.default_rng(seed)
    S, rows_t = sum(table_segments), 900
    tables = [ops.Table(torch.from_numpy(rng.normal(0, 0.1, (rows_t, dim)).astype(np.float32)), table_dtype) for _ in table_segments]
    n = rng.poisson(mean, S) if mean else np.zeros(S, np.int64)
    n[rng.random(S) < 0.1] = 0
    off = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    ids = rng.integers(0, rows_t, int(off[-1]) + tail)
    if len(ids) > 40:
        ids[rng.integers(0, len(ids), 5)] = [-1, rows_t, 1 << 33, (1 << 32) + 5, 0x7fffffff]
    ids, off = torch.from_numpy(ids).cuda(), torch.from_numpy(off).cuda()
    ctx = sharded.ShardContext(0, 1, tables, list(table_segments), dim, max_ids=ids.numel() + 7, partial_dtype=partial)
    rows = S // groups
    one, staged = [torch.full((rows, groups * dim + pad), 9.0, dtype=out_dtype, device="cuda") for _ in range(2)]
    ctx.pool(ids, off, groups, one)
    ctx.begin(ids, off)
    ctx.finish(groups, staged)
    torch.cuda.synchronize()
    assert not ctx.overflow()
    ctx.close()
    assert torch.equal(one[:, groups * dim:], staged[:, groups * dim:])          # the padding stays as it was
    # (+ 0: the combine adds to a positive zero)
    assert torch.equal(one + 0, staged + 0), float((one.float() - staged.float()).abs().max())
    return one


@pytest.mark.parametrize("table_segments,groups,mean", [((1,), 1, 3), ((5, 7), 3, 4), ((6, 6), 4, 60), ((3000, 2000, 0), 5, 9),
                                                        ((30_000, 30_000), 6, 12), ((40_000, 20_001), 9, 1.4), ((64, 64), 2, 0)])
@pytest.mark.parametrize("dim,pad", [(32, 0), (18, 3), (5, 1), (120, 0)])
def test_one_call_equals_the_staged_step(table_segments, groups, mean, dim, pad):
    pkg.load()
    if sum(table_segments) % groups:
        table_segments = table_segments[:-1] + (table_segments[-1] + groups - sum(table_segments) % groups,)
    for table_dtype, partial, out_dtype in ((torch.float16, "f16", torch.float16), (torch.float32, "f32", torch.float32),
                                            (torch.float16, "f32", torch.float16), (torch.float16, "f16", torch.float32)):
        _both(table_segments, groups, mean, dim, table_dtype, partial, out_dtype, pad, 0, 3)


@pytest.mark.parametrize("mean", [2, 9, 70])
def test_ids_past_the_last_offset(mean):
    pkg.load()
    _both((300, 330), 7, mean, 16, torch.float16, "f32", torch.float32, 0, 11, 4)


def test_limits_of_the_one_call_step():
    pkg.load()
    from x_deeplearning_b200 import ops, sharded
    table = ops.Table(torch.zeros((10, 8)), torch.float16)
    ctx = sharded.ShardContext(0, 1, [table], [4], 8, max_ids=5, partial_dtype="f16")
    off = torch.zeros(5, dtype=torch.int32, device="cuda")
    out = torch.zeros((2, 16), dtype=torch.float16, device="cuda")
    with pytest.raises(Exception, match="sized for"):
        ctx.pool(torch.zeros(6, dtype=torch.int64, device="cuda"), off, 2, out)
    with pytest.raises(Exception):
        ctx.pool(torch.zeros(1, dtype=torch.int64, device="cuda"), off, 3, out)             # 4 segments are not 3 groups
    ctx.begin(torch.zeros(1, dtype=torch.int64, device="cuda"), off)
    with pytest.raises(Exception, match="still open"):
        ctx.pool(torch.zeros(1, dtype=torch.int64, device="cuda"), off, 2, out)
    ctx.finish(2, out)
    ctx.close()
