"""Segment offsets of the sharded step made from the received records: runs of empty segments of every length at the start,
in the middle and at the end, few and many records, no records at all."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pattern", ["dense", "sparse", "gaps", "first", "last", "none"])
@pytest.mark.parametrize("B", [1, 70, 5000])
def test_offsets_over_empty_segments(pattern, B):
    pkg.load()
    from x_deeplearning_b200 import ops, sharded
    rng = np.random.default_rng(B + len(pattern))
    nt, gpt, dim, rows = 2, 3, 16, 3000
    S = nt * gpt * B
    n = rng.integers(0, 9, S)
    if pattern == "sparse":
        n[rng.random(S) < 0.97] = 0
    elif pattern == "gaps":
        for at in range(0, S, 61):
            n[at:at + rng.integers(1, 60)] = 0
    elif pattern in ("first", "last"):
        n[:] = 0
        n[0 if pattern == "first" else -1] = 40
    elif pattern == "none":
        n[:] = 0
    w = [torch.from_numpy(rng.normal(0, 0.1, (rows, dim)).astype(np.float16)) for _ in range(nt)]
    tables = [ops.Table(x.float(), torch.float16) for x in w]
    off = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    ids = rng.integers(0, rows, int(off[-1]))
    ctx = sharded.ShardContext(0, 1, tables, [gpt * B] * nt, dim, max_ids=len(ids) + 5, partial_dtype="f32")
    out = torch.full((B, nt * gpt * dim), 9.0, device="cuda")
    for _ in range(3):                                   # both buffer slots, and one of them again
        ctx.pool(torch.from_numpy(ids).cuda(), torch.from_numpy(off).cuda(), nt * gpt, out)
    seg = np.repeat(np.arange(S), n)
    table_of = seg // (gpt * B)
    x = torch.stack([w[t][i].double() for t, i in zip(table_of, ids)]) if len(ids) else torch.zeros((0, dim), dtype=torch.float64)
    want = torch.zeros((S, dim), dtype=torch.float64).index_add_(0, torch.from_numpy(seg), x)
    got = out.view(B, nt * gpt, dim).permute(1, 0, 2).reshape(S, dim).double().cpu()
    assert (got - want).abs().max() <= 40 * 2.0 ** -24 * 40 * 0.5 + 1e-7        # fp32 sums of at most 40 values below 0.5
    assert not ctx.overflow()
    ctx.close()


@pytest.mark.parametrize("segments,mean", [(1, 1), (1, 5000), (300, 3), (9000, 40), (70000, 25), (2_000_000, 0.6)])
def test_routing_to_one_shard(segments, mean):
    """One shard: rows in place, segment numbers found per block of ids (table, or search where most segments are empty)."""
    from cpu_shard_ops import CpuShardOps
    pkg.load()
    from x_deeplearning_b200 import sharded
    rng = np.random.default_rng(segments)
    counts = rng.poisson(mean, segments).astype(np.int32) if segments > 1 else np.array([mean], np.int32)
    if segments == 2_000_000:
        counts[100_000:1_900_000] = 0
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    ids = rng.integers(0, 1 << 40, int(off[-1])).astype(np.int64)
    if len(ids) > 3:
        ids[:3] = [-1, 0, (1 << 50) + 3]
    vals = rng.normal(1, 0.3, len(ids)).astype(np.float32)
    t = torch.from_numpy
    gops, cops = sharded.GpuShardOps(), CpuShardOps()
    for v in (vals, None):
        cv, gv = (None, None) if v is None else (t(v), t(v).cuda())
        for g, c in zip(gops.route(t(ids).cuda(), gv, t(off).cuda(), 1), cops.route(t(ids), cv, t(off), 1)):
            assert torch.equal(g.cpu(), c)
        g, c = gops.route_packed(t(ids).cuda(), gv, t(off).cuda(), 1), cops.route_packed(t(ids), cv, t(off), 1)
        assert torch.equal(g[0].cpu(), c[0]) and torch.equal(g[2].cpu(), c[2])


@pytest.mark.parametrize("sources,cap,S", [(1, 2, 1), (1, 5000, 700), (3, 4099, 6000), (16, 300, 40), (2, 100_000, 3)])
def test_offsets_and_counts_of_received_records(sources, cap, S):
    """The two ways to a source's segments agree: offsets straight from the sorted records (what the sharded step uses) and the
    counts of xb_record_counts_padded added up. Headers that say more than the bucket holds, or less than nothing, and records
    of segments that do not exist (they belong to none)."""
    import ctypes
    pkg.load()
    from x_deeplearning_b200 import capi, ops
    rng = np.random.default_rng(S)
    packed = np.zeros((sources, cap), np.int64)
    want = np.zeros((sources, S), np.int32)
    for s in range(sources):
        cnt = [cap - 1, (cap - 1) // 2, cap + 7, -3, 0][s % 5] if sources > 1 else cap - 1
        real = max(0, min(cnt, cap - 1))
        tags = np.sort(rng.integers(0, S, real)) if s % 2 == 0 else np.sort(rng.integers(S // 3, 1 + S // 2, real) // 5 * 5 % S)
        beyond = min(real, 5) if sources > 1 or cap == 5000 else 0
        if beyond:
            tags[real - beyond:] = S + np.arange(beyond)
            if beyond == 5:
                tags[real - 1] = (1 << 32) - 9                       # the sign bit of the record
        for i, t in enumerate(tags):
            packed[s, 1 + i] = np.uint64((int(t) << 32) | int(rng.integers(0, 1 << 31))).astype(np.int64)
        packed[s, 0] = cnt
        want[s] = np.bincount(tags[tags < S], minlength=S)[:S]
    dp = torch.from_numpy(packed).cuda()
    counts = torch.full((sources, S), -1, dtype=torch.int32, device="cuda")
    offsets = torch.full((sources, S + 1), -1, dtype=torch.int32, device="cuda")
    lib = capi.lib()
    capi.check(lib.xb_record_counts_padded(ops.ptr(dp), sources, cap, ops.ptr(counts), S, ops.stream()))
    fn = lib["_ZN2xb21record_offsets_paddedEPKlilPilP11CUstream_st"]         # xb::record_offsets_padded
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int64, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]
    assert fn(dp.data_ptr(), sources, cap, offsets.data_ptr(), S, ops.stream()) == 0
    assert np.array_equal(counts.cpu().numpy(), want)
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([np.zeros((sources, 1), np.int64), np.cumsum(want, 1)], 1))
