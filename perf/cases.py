"""The work that users of this library give it, as a fixed list of timed cases and a generator of more of them.

Six kinds, each through the entry points a user calls:
  pool       embedding pooling of many feature groups (ops.PoolPlan over xb_embedding_pool)
  sharded    the row-sharded pooling step, one rank (sharded.ShardContext over xb_sharded_pool)
  gemm       parallel branches of a dense layer in one call (ops.gemm over xb_gemm)
  mlp        the layers of a dense tower one after the other (ops.gemm)
  din, dien  a forward pass of the DIN / DIEN-style model on ids in device memory (din.DinModel, dien.DienModel)
  serve      one request batch through blaze::Predictor, host buffers in, probabilities in host memory out
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from __graft_entry__ import load_package  # noqa: E402

load_package()
from x_deeplearning_b200 import blaze_api, capi, dien, din, din_netdef, ops, sharded, workloads  # noqa: E402

_T = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
_UDF = {"sum": capi.XB_UDF_SUM, "avg": capi.XB_UDF_AVG}
_SIZE = {"f16": 2, "bf16": 2, "f32": 4}


def listed():
    return [
        # the sparse features of one small ranking request: hashed feature ids, list lengths as the front end sends
        # them (counts), averages; latency and launches count
        dict(name="pool_request", kind="pool", rows=200_000, dim=18, table="f16", batch=64, groups=12, min_len=0, max_len=20,
             zipf=1.1, hashed=True, counts=True, weighted=True, udf="avg"),
        # the sum-pooling benchmark configuration: 512 samples x 20 feature groups over a 1 M x 16 fp32 table
        dict(name="pool_batch", kind="pool", rows=1_000_000, dim=16, table="f32", batch=512, groups=20, min_len=1, max_len=50,
             zipf=1.1, hashed=False, counts=False, weighted=True, udf="sum"),
        # bulk scoring against one shard of a large table (25 M x 32 fp16, far beyond L2)
        dict(name="pool_bulk", kind="pool", rows=25_000_000, dim=32, table="f16", batch=8192, groups=40, min_len=1, max_len=30,
             zipf=1.05, hashed=False, counts=False, weighted=False, udf="sum"),
        # one rank's step of the row-sharded configuration, scaled to a rank's share of the batch
        dict(name="sharded_step", kind="sharded", tables=4, rows=5_000_000, dim=32, groups=10, batch=8192, max_len=30, zipf=1.05,
             partial="f16"),
        # FusedParallelGemm of a graph as Blaze holds it: one shared input, weights in their [K, N] layout, the branches
        # stacked on axis 0, for the 1000 candidates of a request
        dict(name="gemm_fused_parallel", kind="gemm", P=8, M=1000, N=128, K=256, dtype="f16", layout="kn", shared=True, axis=0,
             act="none"),
        # the parallel-GEMM benchmark configuration: per-branch inputs, packed weights, bias + PReLU, axis-1 concat
        dict(name="gemm_parallel", kind="gemm", P=8, M=4096, N=128, K=256, dtype="f16", layout="packed", shared=False, axis=1,
             act="prelu"),
        # the dense tower of the large-table configuration on a full batch, the compute-bound case
        dict(name="mlp_bulk", kind="mlp", M=65536, dims="1280-1024-512-256-1", dtype="bf16"),
        # one user and a short candidate list: the latency end of DIN serving
        dict(name="din_small", kind="din", requests=1, n_cand=200, T=100, emb=18, h0=80, h1=40, ragged=True, item_rows=200_000),
        # the headline: 74 requests of 1000 candidates
        dict(name="din_bulk", kind="din", requests=74, n_cand=1000, T=100, emb=18, h0=80, h1=40, ragged=False,
             item_rows=5_000_000),
        # DIEN-style model, a batch of requests
        dict(name="dien_batch", kind="dien", requests=16, n_cand=1000, T=100, emb=18, h0=80, h1=40, ragged=False,
             item_rows=200_000),
        # one serving request end to end from host buffers: fp16 model, fused graph
        dict(name="serve_f16", kind="serve", requests=1, n_cand=1000, T=100, form="fused"),
        # the same model as the reference runs it: an fp32 graph of the reference's own operators
        dict(name="serve_f32", kind="serve", requests=1, n_cand=500, T=100, form="reference_f32"),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["pool", "pool", "sharded", "gemm", "gemm", "mlp", "din", "din", "dien", "serve"])
    if kind == "pool":
        table = rng.choice(["f16", "f32"])
        groups, max_len = rng.randint(1, 40), _log(rng, 1, 100)
        batch = _log(rng, 1, min(65536, 10_000_000 // (groups * (max_len + 1))))
        hashed = rng.random() < 0.4
        return dict(kind="pool", rows=_log(rng, 1000, 500_000 if hashed else 20_000_000), dim=rng.choice([4, 8, 12, 16, 18, 32, 36, 64]),
                    table=table, batch=batch, groups=groups, min_len=rng.choice([0, 1]), max_len=max_len,
                    zipf=rng.choice([1.05, 1.1]), hashed=hashed, counts=rng.random() < 0.5, weighted=rng.random() < 0.5,
                    udf=rng.choice(["sum", "avg"]))
    if kind == "sharded":
        return dict(kind="sharded", tables=rng.randint(1, 4), rows=_log(rng, 10_000, 5_000_000), dim=rng.choice([8, 16, 32, 64]),
                    groups=rng.randint(1, 10), batch=_log(rng, 64, 8192), max_len=_log(rng, 1, 30), zipf=1.05,
                    partial=rng.choice(["f16", "f32"]))
    if kind == "gemm":
        dtype = rng.choice(["f16", "f16", "bf16", "f32"])
        P, K, N = rng.choice([1, 2, 4, 8, 16]), _log(rng, 16, 512), _log(rng, 8, 512)
        if rng.random() < 0.75:
            K, N = (K + 7) // 8 * 8, (N + 7) // 8 * 8
        M = _log(rng, 16, min(65536, int((4e9 if dtype == "f32" else 3e10) / (P * K * N))))
        return dict(kind="gemm", P=P, M=M, N=N, K=K, dtype=dtype, layout="kn" if dtype == "f32" else rng.choice(["kn", "packed"]),
                    shared=rng.random() < 0.5, axis=rng.choice([0, 1]), act=rng.choice(["none", "prelu", "dice", "sigmoid"]))
    if kind == "mlp":
        dims = rng.choice(["1280-1024-512-256-1", "640-512-256-1", "328-200-80-2", "288-256-128-2", "1024-1024-1024"])
        return dict(kind="mlp", M=_log(rng, 32, 65536), dims=dims, dtype=rng.choice(["f16", "bf16"]))
    if kind == "serve":
        form = rng.choice(["fused", "fused", "reference_f32"])
        if form == "fused":
            return dict(kind="serve", requests=_log(rng, 1, 8), n_cand=_log(rng, 20, 1000), T=rng.choice([20, 50, 100]), form=form)
        return dict(kind="serve", requests=1, n_cand=_log(rng, 20, 500), T=rng.choice([20, 50, 100]), form=form)
    h0, h1 = rng.choice([(80, 40), (80, 40), (64, 32)])
    c = dict(kind=kind, n_cand=_log(rng, 20, 1000), T=rng.choice([20, 50, 77, 100]), emb=rng.choice([18, 18, 16]), h0=h0, h1=h1,
             ragged=rng.random() < 0.5, item_rows=_log(rng, 10_000, 1_000_000))
    c["requests"] = _log(rng, 1, 74 if kind == "din" else 16 if c["emb"] == 18 else 4)
    return c


# ---- inputs -------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _zipf(g, rows, n, s):
    """n row numbers, rank r with probability ~ 1/(r+1)^s (continuous power-law inverse), hot rows spread over the table."""
    a = 1.0 - s
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    r = (u * ((rows + 1.0) ** a - 1.0) + 1.0) ** (1.0 / a) - 1.0
    ranks = r.to(torch.int64).clamp_(0, rows - 1)
    mult = 2654435761 % rows
    while np.gcd(mult, rows) != 1:
        mult += 1
    return (ranks * mult + 12345) % rows


def _device_table(g, rows, dim, dtype, keys=None):
    """An ops.Table whose image is made in device memory (its constructor takes a host image)."""
    tb = ops.Table.__new__(ops.Table)
    es = _SIZE[dtype]
    code = capi.XB_F16 if dtype == "f16" else capi.XB_F32
    pitch = int(capi.lib().xb_table_row_pitch(dim, code))
    tb.rows, tb.dim, tb.dtype, tb.pitch = rows, dim, _T[dtype], pitch
    tb.buf = torch.empty((rows, pitch // es), dtype=_T[dtype], device="cuda").normal_(0, 0.1, generator=g)
    tb.buf[:, dim:] = 0
    tb.desc = capi.TableDesc()
    tb.desc.weights, tb.desc.rows, tb.desc.dim, tb.desc.dtype, tb.desc.row_pitch_bytes = tb.buf.data_ptr(), rows, dim, code, pitch
    tb.slot_keys = tb.slot_rows = None
    if keys is not None:
        slots = 16
        while slots < 2 * rows:
            slots <<= 1
        sk, sr = torch.empty(slots, dtype=torch.int64), torch.empty(slots, dtype=torch.int32)
        capi.check(capi.lib().xb_table_build_index_host(ops.ptr(keys), rows, slots, ops.ptr(sk), ops.ptr(sr)))
        tb.slot_keys, tb.slot_rows = sk.cuda(), sr.cuda()
        tb.desc.slot_keys, tb.desc.slot_rows, tb.desc.slots = tb.slot_keys.data_ptr(), tb.slot_rows.data_ptr(), slots
    return tb


def _prepare_pool(c, seed):
    g = _gen(seed)
    keys = None
    if c["hashed"]:
        # 64-bit feature hashes: an odd multiplier makes the map from row numbers one to one
        keys = (torch.arange(c["rows"], dtype=torch.int64) + 1) * -7046029254386353131
    table = _device_table(g, c["rows"], c["dim"], c["table"], keys)
    dkeys = keys.cuda() if keys is not None else None
    B, G, dim = c["batch"], c["groups"], c["dim"]
    out = torch.zeros((B, G * dim), dtype=_T[c["table"]], device="cuda")
    groups = []
    for i in range(G):
        counts = torch.randint(c["min_len"], c["max_len"] + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
        n = int(counts.sum())
        ids = _zipf(g, c["rows"], n, c["zipf"])
        if dkeys is not None:
            ids = dkeys[ids]
            ids[torch.rand(n, generator=g, device="cuda") < 0.02] = 12345        # features the table has not seen
        values = torch.rand(n, generator=g, device="cuda") + 0.5 if c["weighted"] else None
        if c["counts"]:
            segs = counts
        else:
            segs = torch.zeros(B + 1, dtype=torch.int32, device="cuda")
            torch.cumsum(counts, 0, dtype=torch.int32, out=segs[1:])
        groups.append(ops.make_group(table, ids, values, segs, [dict(udf=_UDF[c["udf"]], out=out, col=i * dim)], _T[c["table"]],
                                     segments_are_offsets=not c["counts"]))
    return dict(c, plan=ops.PoolPlan(groups), groups=groups, out=out)


def _run_pool(s):
    s["plan"].run()
    return s["out"]


class _Closing:
    """Calls `close` of what it holds when the state that holds it goes away."""

    def __init__(self, *things):
        self.things = things

    def __del__(self):
        if not sys.is_finalizing():
            for t in self.things:
                t.close()


def _prepare_sharded(c, seed):
    g = _gen(seed)
    B, nt, gpt = c["batch"], c["tables"], c["groups"]
    tables = [_device_table(g, c["rows"], c["dim"], "f16") for _ in range(nt)]
    counts = torch.randint(1, c["max_len"] + 1, (nt * gpt * B,), generator=g, device="cuda", dtype=torch.int32)
    off = torch.zeros(len(counts) + 1, dtype=torch.int32, device="cuda")
    torch.cumsum(counts, 0, dtype=torch.int32, out=off[1:])
    ids = _zipf(g, c["rows"], int(off[-1]), c["zipf"])
    ctx = sharded.ShardContext(0, 1, tables, [gpt * B] * nt, c["dim"], ids.numel() + 4096, c["partial"], capacity_factor=1.2)
    out = torch.zeros((B, nt * gpt * c["dim"]), dtype=_T[c["partial"]], device="cuda")
    return dict(c, ctx=ctx, closing=_Closing(ctx), ids=ids, off=off, out=out, keep=tables)


def _run_sharded(s):
    return s["ctx"].pool(s["ids"], s["off"], s["tables"] * s["groups"], s["out"])


def _prepare_gemm(c, seed):
    g = _gen(seed)
    P, M, N, K, dt = c["P"], c["M"], c["N"], c["K"], _T[c["dtype"]]
    r = lambda *sh: torch.randn(sh, generator=g, device="cuda")
    A = r(*((M, K) if c["shared"] else (P, M, K))).to(dt)
    W = (r(P, K, N) / K ** 0.5).to(dt)
    s = dict(c, A=A, W_in=W, bias=r(P, N) * 0.1)
    kw = dict(batch=P, M=M, N=N, K=K, lda=K, bias_kind=capi.XB_BIAS_ROW)
    if c["layout"] == "packed":
        # constants are laid out once when a model is loaded
        s["W"] = ops.pack_weight_kmajor(W if P > 1 else W[0], dt, batch=P)
        kw.update(trans_b=True, ldb=s["W"].shape[-1])
        stride_b = N * s["W"].shape[-1]
    else:
        s["W"] = W
        kw.update(trans_b=False, ldb=N)
        stride_b = K * N
    if c["axis"] == 1:
        s["Y"] = torch.zeros((M, P * N), dtype=dt, device="cuda")
        kw.update(ldy=P * N, strides=(0 if c["shared"] else M * K, stride_b, N, N))
    else:
        s["Y"] = torch.zeros((P * M, N), dtype=dt, device="cuda")
        kw.update(ldy=N, strides=(0 if c["shared"] else M * K, stride_b, N, M * N))
    if c["act"] == "prelu":
        kw.update(epilogue=capi.XB_EPI_PRELU, ep=(torch.full((1,), 0.25, device="cuda"), None, None), ep_count=1)
    elif c["act"] == "dice":
        u = lambda lo, hi: torch.rand((P, N), generator=g, device="cuda") * (hi - lo) + lo
        kw.update(epilogue=capi.XB_EPI_DICE, ep=(u(0, 0.5), u(-0.1, 0.1), u(0.5, 1.5)), stride_ep=N)
    elif c["act"] == "sigmoid":
        kw.update(epilogue=capi.XB_EPI_SIGMOID)
    s["kw"] = kw
    return s


def _run_gemm(s):
    return ops.gemm(s["A"], s["W"], Y=s["Y"], bias=s["bias"], **s["kw"])


def _prepare_mlp(c, seed):
    g = _gen(seed)
    dims, dt, M = [int(x) for x in c["dims"].split("-")], _T[c["dtype"]], c["M"]
    r = lambda *sh: torch.randn(sh, generator=g, device="cuda")
    layers = []
    for i, (k, n) in enumerate(zip(dims, dims[1:])):
        last = i == len(dims) - 2
        act = dict(epilogue=capi.XB_EPI_SIGMOID) if last else dict(
            epilogue=capi.XB_EPI_PRELU, ep=(torch.full((1,), 0.25, device="cuda"), None, None), ep_count=1)
        layers.append(dict(W=(r(n, k) / k ** 0.5).to(dt), bias=r(n) * 0.1, Y=torch.zeros((M, n), dtype=dt, device="cuda"),
                           kw=dict(trans_b=True, M=M, N=n, K=k, **act)))
    return dict(c, x=r(M, dims[0]).to(dt), layers=layers)


def _run_mlp(s):
    x, ys = s["x"], []
    for y in s["layers"]:
        x = ops.gemm(x, y["W"], Y=y["Y"], bias=y["bias"], **y["kw"])
        ys.append(x)
    return ys


def _model(c, seed, make):
    """workloads' random-init model with the case's sizes; the item table is made on the device, where that is quick."""
    D = workloads.DIN_DIMS
    keep = dict(D)
    try:
        D.update(emb=c.get("emb", 18), d=2 * c.get("emb", 18), T=c["T"], h0=c.get("h0", 80), h1=c.get("h1", 40))
        m = make(seed, item_rows=1000, cate_rows=10_000, user_rows=10_000, emb_sigma=0.5)
    finally:
        D.clear()
        D.update(keep)
    rows = c.get("item_rows", 200_000)
    item = torch.empty((rows, m["dims"]["emb"]), dtype=torch.float16, device="cuda").normal_(0, 0.5, generator=_gen(seed))
    m["item"] = item.cpu().float().numpy()
    m["dims"]["item_rows"] = rows
    return m


def _requests(m, c, seed):
    g, D, R, n, T = _gen(seed + 1), m["dims"], c["requests"], c["n_cand"], c["T"]
    z = lambda rows, k: _zipf(g, rows, k, 1.1).cpu().numpy()
    seq = torch.randint(1, T + 1, (R,), generator=g, device="cuda").cpu().numpy() if c.get("ragged") else np.full(R, T)
    h = int(seq.sum())
    return dict(requests=R, n_cand=n, T=T, seq_len=seq.astype(np.int32),
                user_ids=np.stack([z(D["user_rows"], R) for _ in range(D["user_groups"])], 1), hist_item=z(D["item_rows"], h),
                hist_cate=z(D["cate_rows"], h), cand_item=z(D["item_rows"], R * n), cand_cate=z(D["cate_rows"], R * n))


def _prepare_din(c, seed):
    m = _model(c, seed, workloads.din_model if c["kind"] == "din" else workloads.dien_model)
    net = (din.DinModel if c["kind"] == "din" else dien.DienModel)(m)
    return dict(c, net=net, p=net.upload(net.stage(_requests(m, c, seed))))


def _run_din(s):
    if s["kind"] == "din":
        return s["net"].forward_device(s["p"])
    prob, inner = s["net"].forward_dien(s["p"])
    return prob, inner["hseq"], inner["scores"], inner["final"]


def _prepare_serve(c, seed):
    m = _model(c, seed, workloads.din_model)
    fused = c["form"] == "fused"
    if fused:
        text, _ = din_netdef.build(m)
    else:
        text, _ = din_netdef.build_unfused(m, dtype=capi.XB_F32, device_type=1)
    mgr = blaze_api.PredictorManager()
    din_netdef.register_tables(mgr, m)
    mgr.load_model_text(text, optimize=True)
    pred = mgr.create_predictor(device_type=1, device_id=torch.cuda.current_device())
    feeds = {}
    for n, a in din_netdef.feeds_of(m, _requests(m, c, seed)).items():
        if n.endswith(".values") and not fused:
            a = a.astype(np.float32)
        feeds[n] = torch.from_numpy(a).pin_memory().numpy()
    out = torch.empty((c["requests"] * c["n_cand"], 2), dtype=torch.float32).pin_memory().numpy()
    return dict(c, pred=pred, closing=_Closing(pred, mgr), feeds=feeds, out=out)


def _run_serve(s):
    pred = s["pred"]
    for n, a in s["feeds"].items():
        pred.feed(n, a)
    pred.forward()
    return pred.output("output", into=s["out"])


_KINDS = {"pool": (_prepare_pool, _run_pool), "sharded": (_prepare_sharded, _run_sharded), "gemm": (_prepare_gemm, _run_gemm),
          "mlp": (_prepare_mlp, _run_mlp), "din": (_prepare_din, _run_din), "dien": (_prepare_din, _run_din),
          "serve": (_prepare_serve, _run_serve)}


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return _KINDS[state["kind"]][1](state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------
def _pool_bytes(rows, dim, es, segments, n, per_id, out_es):
    return int(n * per_id + min(n, rows) * dim * es + segments * 4 + segments * dim * out_es)


def work(case):
    c = case
    if c["kind"] == "pool":
        es, segs = _SIZE[c["table"]], c["batch"] * c["groups"]
        n = segs * (c["min_len"] + c["max_len"]) / 2
        return {"bytes": _pool_bytes(c["rows"], c["dim"], es, segs, n, 12 if c["weighted"] else 8, es), "flops": 2 * n * c["dim"]}
    if c["kind"] == "sharded":
        segs = c["tables"] * c["groups"] * c["batch"]
        n = segs * (1 + c["max_len"]) / 2
        return {"bytes": _pool_bytes(c["tables"] * c["rows"], c["dim"], 2, segs, n, 8, _SIZE[c["partial"]]), "flops": 2 * n * c["dim"]}
    if c["kind"] == "gemm":
        P, M, N, K = c["P"], c["M"], c["N"], c["K"]
        return {"bytes": _SIZE[c["dtype"]] * ((1 if c["shared"] else P) * M * K + P * K * N + P * M * N), "flops": 2 * P * M * N * K}
    if c["kind"] == "mlp":
        d = [int(x) for x in c["dims"].split("-")]
        w = sum(a * b for a, b in zip(d, d[1:]))
        return {"bytes": 2 * (c["M"] * sum(d) + w), "flops": 2 * c["M"] * w}
    # the models: ids in, table rows once per id, probabilities out; the multiply-adds of the dense layers
    e, h0, h1 = c.get("emb", 18), c.get("h0", 80), c.get("h1", 40)
    d, R, N, T = 2 * e, c["requests"], c["requests"] * c["n_cand"], c["T"]
    t = T * (1 + T) / (2 * T) if c.get("ragged") else T
    ids = 8 * R + 2 * R * t + 2 * N
    bytes_ = ids * (8 + 2 * e) + 8 * N
    flops = 2 * N * T * (4 * d * h0 + h0 * h1 + h1) + 2 * N * (8 * e * 200 + 5 * d * 200 + 200 * 80 + 160)
    if c["kind"] == "dien":
        # GRU states, scores and final states are results too
        bytes_ += 2 * R * T * d + 4 * N * T + 2 * N * d
        flops += 2 * R * T * 6 * d * d + 2 * N * T * 3 * d * d
    else:
        flops += 2 * N * T * d
    return {"bytes": int(bytes_), "flops": int(flops)}


def tolerance(case):
    """About four times the 2-norm difference between the path and a float64 restatement of it, on listed and drawn cases:
    6.6e-8 for fp32 sums over id lists, 2.3e-7 for fp32 products, 2.1e-4 / 1.7e-3 where one fp16 / bf16 rounding of the result
    decides, 2.0e-3 for a chain of bf16 layers, 4.7e-4 for the DIN probabilities and 6.3e-4 for the states of the DIEN model."""
    c = case
    if c["kind"] in ("pool", "sharded"):
        return {"rel": 5e-7 if c.get("table", c.get("partial")) == "f32" else 8e-4}
    if c["kind"] in ("gemm", "mlp"):
        return {"rel": {"f32": 1e-6, "f16": 9e-4, "bf16": 8e-3}[c["dtype"]]}
    if c["kind"] == "serve":
        return {"rel": 1e-6 if c["form"] == "reference_f32" else 2e-3}
    return {"rel": 2e-3 if c["kind"] == "din" else 2.5e-3}


# ---- the same results in 64 bits, by plain torch ----------------------------------------------------------------
_INVERSE = pow(-7046029254386353131, -1, 1 << 64)
_INVERSE -= (_INVERSE >> 63) << 64                                   # as a signed 64-bit number


def _exact_pool(c, seed):
    s = _prepare_pool(c, seed)
    out = torch.zeros((c["batch"], c["groups"], c["dim"]), dtype=torch.float64, device="cuda")
    for i, grp in enumerate(s["groups"]):
        table, ids, values, segs, _ = grp._keep
        lens = segs.long() if c["counts"] else segs.long().diff()
        # a hashed key is (row + 1) * multiplier, undone by the multiplier's inverse; what gives no row is not in the table
        row = ids * _INVERSE - 1 if c["hashed"] else ids
        known = (row >= 0) & (row < c["rows"])
        seg = torch.repeat_interleave(torch.arange(c["batch"], device="cuda"), lens)[known]
        x = table.buf[row[known], :c["dim"]].double()
        if values is not None:
            x *= values[known].double()[:, None]
        out[:, i].index_add_(0, seg, x)
        if c["udf"] == "avg":
            out[:, i] /= lens.clamp(min=1)[:, None]
    return out.view(c["batch"], -1)


def _exact_sharded(c, seed):
    s = _prepare_sharded(c, seed)
    B, gpt = c["batch"], c["groups"]
    off = s["off"].long()
    out = torch.zeros((B, c["tables"] * gpt, c["dim"]), dtype=torch.float64, device="cuda")
    for slot in range(c["tables"] * gpt):
        o = off[slot * B:(slot + 1) * B + 1]
        x = s["keep"][slot // gpt].buf[s["ids"][o[0]:o[-1]], :c["dim"]].double()
        out[:, slot].index_add_(0, torch.repeat_interleave(torch.arange(B, device="cuda"), o.diff()), x)
    return out.view(B, -1)


def _exact_gemm(c, seed):
    s = _prepare_gemm(c, seed)
    y = torch.matmul(s["A"].double(), s["W_in"].double()) + s["bias"].double()[:, None]
    if c["act"] == "prelu":
        y = torch.where(y < 0, y * 0.25, y)
    elif c["act"] == "dice":
        y = _dice(y, *[t.double()[:, None] for t in s["kw"]["ep"]])
    elif c["act"] == "sigmoid":
        y = y.sigmoid()
    return y.permute(1, 0, 2).reshape(c["M"], -1) if c["axis"] == 1 else y.reshape(-1, c["N"])


def _exact_mlp(c, seed):
    s = _prepare_mlp(c, seed)
    x, ys = s["x"].double(), []
    for i, y in enumerate(s["layers"]):
        x = x @ y["W"].double().t() + y["bias"].double()
        x = x.sigmoid() if i == len(s["layers"]) - 1 else torch.where(x < 0, x * 0.25, x)
        ys.append(x)
    return ys


def _dice(x, gamma, mean, var):
    p = ((x - mean) / (var + 1e-8).sqrt()).sigmoid()
    return (1 - p) * gamma * x + p * x


def _exact_model(c, seed):
    """The model op by op: embeddings, (GRU,) attention unit, (AUGRU,) tower, softmax."""
    dien_ = c["kind"] == "dien"
    m = _model(c, seed, workloads.dien_model if dien_ else workloads.din_model)
    req, D = _requests(m, c, seed), m["dims"]
    D64 = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda").double()
    rows = lambda w, ids: D64(w[ids])
    R, n, T, d = c["requests"], c["n_cand"], c["T"], D["d"]
    user = torch.cat([rows(m["user"][g], req["user_ids"][:, g]) for g in range(D["user_groups"])], 1)
    hist = torch.cat([rows(m["item"], req["hist_item"]), rows(m["cate"], req["hist_cate"])], 1)
    q = torch.cat([rows(m["item"], req["cand_item"]), rows(m["cate"], req["cand_cate"])], 1)
    k = torch.zeros((R, T, d), dtype=torch.float64, device="cuda")
    at = 0
    for r, ln in enumerate(req["seq_len"].tolist()):                # lists end at the last step
        k[r, T - ln:] = hist[at:at + ln]
        at += ln
    W = lambda group: {x: D64(v) for x, v in m[group].items()}
    a = W("att")
    tw = {x: [D64(y) for y in v] if isinstance(v, tuple) else D64(v) for x, v in m["dien_tower" if dien_ else "tower"].items()}
    h = _exact_gru(k, W("gru")) if dien_ else k
    act = (lambda x, i: x.sigmoid()) if dien_ else (lambda x, i: _dice(x, a["g" + i], a["m" + i], a["v" + i]))
    scores = torch.empty((R * n, T), dtype=torch.float64, device="cuda")
    for r in range(R):
        qr, kr = q[r * n:(r + 1) * n, None].expand(n, T, d), h[r][None].expand(n, T, d)
        y = act(torch.cat([qr, kr, qr - kr, qr * kr], 2) @ a["W0"] + a["b0"], "0")
        scores[r * n:(r + 1) * n] = (act(y @ a["W1"] + a["b1"], "1") @ a["W2"] + a["b2"])[..., 0]
    if dien_:
        scores = scores.softmax(1)
        att = _exact_augru(h, scores, n, W("augru"))
    else:
        att = torch.bmm(scores.view(R, n, T), k).view(R * n, d)
    wide = lambda x: x.repeat_interleave(n, 0)
    his = wide(k.sum(1))
    x = torch.cat([wide(user), q, his, q * his, att] + ([] if dien_ else [q - his]), 1)
    for i in "12":
        x = x @ tw["W" + i] + tw["b" + i]
        x = torch.where(x < 0, x * tw["slope" + i], x) if dien_ else _dice(x, *tw["dice" + i])
    prob = (x @ tw["W3"] + tw["b3"]).softmax(1)
    if c["kind"] == "serve":
        return prob.cpu().numpy()
    return (prob, h.reshape(R, T * d), scores, att) if dien_ else prob


def _exact_gru(x, g):
    R, T, H = x.shape
    h, ys = torch.zeros((R, H), dtype=torch.float64, device="cuda"), []
    begun = torch.zeros((R, 1), dtype=torch.bool, device="cuda")
    for t in range(T):
        i = x[:, t] @ g["i2h"]
        begun |= (i[:, :H] != 0).any(1, keepdim=True)               # zero steps in front of a list leave the state at zero
        i, a = i + g["i2h_bias"], h @ g["h2h"] + g["h2h_bias"]
        r, z = (i + a)[:, :2 * H].sigmoid().split(H, 1)
        cand = torch.tanh(i[:, 2 * H:] + r * a[:, 2 * H:])
        h = torch.where(begun, cand + z * (h - cand), 0.0)
        ys.append(h)
    return torch.stack(ys, 1)


def _exact_augru(x, scores, n, g):
    R, T, H = x.shape
    h = torch.zeros((R * n, H), dtype=torch.float64, device="cuda")
    for t in range(T):
        xt = x[:, t].repeat_interleave(n, 0)
        r, u = (torch.cat([xt, h], 1) @ g["Wg"] + g["bg"]).sigmoid().split(H, 1)
        cand = torch.tanh(torch.cat([xt, r * h], 1) @ g["Wc"] + g["bc"])
        u = (1 - scores[:, t:t + 1]) * u
        h = u * h + (1 - u) * cand
    return h


def exact(case, seed):
    return {"pool": _exact_pool, "sharded": _exact_sharded, "gemm": _exact_gemm, "mlp": _exact_mlp}.get(
        case["kind"], _exact_model)(case, seed)
