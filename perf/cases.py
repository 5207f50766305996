"""Timing cases of the engine's public entry points.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (an index with its rows added, queries, result buffers), `run` is one
call, `work` the bytes and operations the call cannot do without and `exact`
the distances in 64 bits, from plain torch.

Kinds of case:

* ``search``: ``IndexBF.search`` on a resident index, with CUDA tensors or, with
  ``host``, numpy arrays;
* ``one_shot``: ``search_l2_distance``, which takes the rows themselves;
* ``batch``: ``SearchBatch.run``, many uneven query batches over several indexes;
* ``serve``: a burst of requests through ``Server`` with pinned host buffers.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import curplsh_b200 as cb
from curplsh_b200 import synth

EXACT, BF16, FP8 = cb.Precision.FP32_EXACT, cb.Precision.BF16_RERANK, cb.Precision.FP8_RERANK
DIMS = (64, 96, 100, 101, 128, 200, 256, 384, 512, 960)


def listed():
    return [
        # one query of an interactive program against a small table: call latency
        {"name": "one_query", "kind": "search", "form": EXACT, "data": "uniform",
         "n": 10_000, "q": 1, "d": 128, "k": 10, "host": False},
        # the plain small configuration: 10,000 uniform rows, 100 queries
        {"name": "uniform_small", "kind": "search", "form": EXACT, "data": "uniform",
         "n": 10_000, "q": 100, "d": 128, "k": 10, "host": False},
        # a handful of queries against a large table: the database is read once
        {"name": "few_queries", "kind": "search", "form": BF16, "data": "bf16",
         "n": 2_000_000, "q": 16, "d": 128, "k": 10, "host": False},
        # host arrays in and out, odd sizes, rows that are no multiple of 16 bytes
        {"name": "ragged_host", "kind": "search", "form": EXACT, "data": "uniform",
         "n": 123_457, "q": 777, "d": 101, "k": 37, "host": True},
        # the integer mixture at full size in both of its forms
        {"name": "mixture_bf16", "kind": "search", "form": BF16, "data": "integers",
         "n": 1_000_000, "q": 10_000, "d": 128, "k": 100, "host": False},
        {"name": "mixture_exact", "kind": "search", "form": EXACT, "data": "integers",
         "n": 1_000_000, "q": 10_000, "d": 128, "k": 100, "host": False},
        # the precision form at scale: unit-sphere rows in FP8
        {"name": "sphere_fp8", "kind": "search", "form": FP8, "data": "sphere",
         "n": 10_000_000, "q": 10_000, "d": 96, "k": 10, "host": False},
        # long result lists (the largest k the engine takes)
        {"name": "large_k", "kind": "search", "form": EXACT, "data": "uniform",
         "n": 300_000, "q": 1_000, "d": 64, "k": 1024, "host": False},
        # wide rows (image descriptors such as GIST's 960 columns)
        {"name": "wide_rows", "kind": "search", "form": BF16, "data": "bf16",
         "n": 200_000, "q": 2_000, "d": 960, "k": 50, "host": False},
        # rows given with the call: they are prepared, searched once and dropped
        {"name": "one_shot", "kind": "one_shot", "form": EXACT, "data": "uniform",
         "n": 200_000, "q": 1_000, "d": 128, "k": 10},
        # 64 uneven batches over 8 resident indexes in one graph replay
        {"name": "batched_uneven", "kind": "batch", "form": EXACT, "spec": 3, "dbs": 8, "batches": 64,
         "n_hi": 2_000_000, "q_hi": 4096},
        # a backlog of 64 requests of 1-256 queries on the serving loop
        {"name": "serving_burst", "kind": "serve", "form": BF16, "data": "bf16",
         "n": 5_000_000, "d": 256, "k": 50, "requests": 64, "sizes": 17},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("search",) * 8 + ("one_shot", "batch", "serve"))
    if kind == "batch":
        return {"kind": "batch", "form": EXACT, "spec": rng.randrange(1 << 20), "dbs": rng.randint(2, 6),
                "batches": rng.randint(8, 40), "n_hi": log_int(50_000, 500_000), "q_hi": log_int(128, 2048)}
    if kind == "serve":
        return {"kind": "serve", "form": BF16, "data": "bf16", "n": log_int(200_000, 4_000_000),
                "d": rng.choice((64, 128, 256)), "k": log_int(1, 100), "requests": log_int(4, 64),
                "sizes": rng.randrange(1 << 20)}
    if kind == "one_shot":
        return {"kind": "one_shot", "form": EXACT, "data": "uniform", "n": log_int(10_000, 500_000),
                "q": log_int(1, 4096), "d": rng.choice(DIMS[:7]), "k": log_int(1, 128)}
    form = rng.choice((EXACT, BF16, FP8))
    while True:
        n, q = log_int(10_000, {EXACT: 2_000_000, BF16: 5_000_000, FP8: 10_000_000}[form]), log_int(1, 10_000)
        d, k = rng.choice(DIMS), log_int(1, {EXACT: 1024, BF16: 256, FP8: 100}[form])
        if q * k <= 1_000_000 and (q + 128) * n * d * (3 if form == EXACT else 1) <= 5e12 and n * d <= 1_000_000_000:
            break
    data = {EXACT: ("uniform", "integers"), BF16: ("integers", "bf16"), FP8: ("sphere",)}[form]
    return {"kind": "search", "form": form, "data": rng.choice(data), "n": n, "q": q, "d": d, "k": k,
            "host": rng.random() < 0.2}


# ---------------------------------------------------------------- inputs
def _bf16(x):
    return x.to(torch.bfloat16).to(torch.float32)


def _rows(gen, data, n, d, cent):
    """n rows of a distribution on the GPU (FP32); `cent` are its centroids."""
    dev = gen.device
    if data == "uniform":
        return torch.rand((n, d), generator=gen, device=dev)
    if data == "normal":
        return _bf16(torch.randn((n, d), generator=gen, device=dev))
    out = torch.empty((n, d), device=dev)
    step = max(1, (1 << 28) // d)
    for a in range(0, n, step):
        m = min(step, n - a)
        x = torch.randn((m, d), generator=gen, device=dev)
        x *= {"integers": 12.0, "sphere": 0.05, "bf16": 0.25}[data]
        x += cent[torch.randint(cent.shape[0], (m,), generator=gen, device=dev)]
        if data == "integers":
            x.round_().clamp_(0.0, 255.0)
        elif data == "sphere":
            x /= x.norm(dim=1, keepdim=True)
        else:
            x = _bf16(x)
        out[a:a + m] = x
    return out


def _table(case, seed, queries):
    """(rows, queries) of one table."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    d, data, cent = case["d"], case["data"], None
    if data == "integers":
        cent = torch.rand((1000, d), generator=gen, device="cuda") * 255.0
    elif data == "sphere":
        cent = torch.randn((4096, d), generator=gen, device="cuda")
        cent = cent / cent.norm(dim=1, keepdim=True)
    elif data == "bf16":
        cent = torch.randn((2048, d), generator=gen, device="cuda")
    return _rows(gen, data, case["n"], d, cent), _rows(gen, data, queries, d, cent)


def _sizes(case):
    """Request sizes of a burst: 1-256 queries, log-uniform."""
    r = random.Random(case["sizes"])
    return [int(round(math.exp(r.uniform(0.0, math.log(256))))) for _ in range(case["requests"])]


def _spec(case):
    dbs, batches = synth.batched_uneven_spec(seed=case["spec"], num_dbs=case["dbs"], num_batches=case["batches"],
                                             n_hi=case["n_hi"], q_hi=case["q_hi"])
    return dbs, batches


def _batch_inputs(case, seed):
    """Rows of every index, and the queries of every batch."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dbs, batches = _spec(case)
    rows = [_rows(gen, "normal", n, d, None) for n, d in dbs]
    return rows, [_rows(gen, "normal", nq, dbs[db][1], None) for db, nq, _ in batches]


def _index(res, rows, form):
    torch.cuda.synchronize()  # add() does not wait for the streams the rows come from
    ix = cb.IndexBF(res, rows.shape[1], cb.IndexBFConfig(device=0, precision=form))
    ix.add(rows.shape[0], rows)
    return ix


def _split(flat, shapes):
    """Contiguous views of a flat buffer."""
    out, at = [], 0
    for m, k in shapes:
        out.append(flat[at:at + m * k].view(m, k))
        at += m * k
    return out


def prepare(case, seed):
    kind = case["kind"]
    res = cb.DeviceResources(0)
    s = {"kind": kind, "res": res}
    if kind == "batch":
        rows, queries = _batch_inputs(case, seed)
        s["indexes"] = [_index(res, x, case["form"]) for x in rows]
        shapes = [(nq, k) for _, nq, k in _spec(case)[1]]
        total = sum(m * k for m, k in shapes)
        s["idx"] = torch.empty(total, dtype=torch.int32, device="cuda")
        s["dist"] = torch.empty(total, device="cuda")
        items = [(s["indexes"][db], q, k, i, x) for (db, _, k), q, i, x in
                 zip(_spec(case)[1], queries, _split(s["idx"], shapes), _split(s["dist"], shapes))]
        s["batch"] = cb.SearchBatch(items)
        return s
    if kind == "serve":
        sizes = _sizes(case)
        k = s["k"] = case["k"]
        rows, queries = _table(case, seed, sum(sizes))
        s["index"] = _index(res, rows, case["form"])
        s["server"] = cb.Server(s["index"])
        s["queries"] = queries.cpu().pin_memory().split(sizes)
        s["idx"] = torch.empty(sum(sizes) * k, dtype=torch.int32).pin_memory()
        s["dist"] = torch.empty(sum(sizes) * k).pin_memory()
        shapes = [(m, k) for m in sizes]
        s["requests"] = list(zip(s["queries"], _split(s["idx"], shapes), _split(s["dist"], shapes)))
        return s
    q, k = case["q"], case["k"]
    rows, queries = _table(case, seed, q)
    s["k"] = k
    if kind == "one_shot":
        s["rows"], s["queries"] = rows, queries
    else:
        s["index"] = _index(res, rows, case["form"])
        s["queries"] = queries.cpu().numpy() if case["host"] else queries
    if case.get("host"):
        s["idx"], s["dist"] = np.empty((q, k), np.int32), np.empty((q, k), np.float32)
    else:
        s["idx"] = torch.empty((q, k), dtype=torch.int32, device="cuda")
        s["dist"] = torch.empty((q, k), device="cuda")
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "search":
        s["index"].search(s["queries"].shape[0], s["queries"], s["k"], s["idx"], s["dist"])
    elif kind == "one_shot":
        cb.search_l2_distance(s["res"], s["rows"], None, s["queries"], s["k"], s["idx"], s["dist"], True)
    elif kind == "batch":
        s["batch"].run()
    else:
        server, k = s["server"], s["k"]
        tickets = [server.submit(q, k, i, x) for q, i, x in s["requests"]]
        for t in tickets:
            server.wait(t)
    return {"distances": s["dist"], "indices": s["idx"]}


def work(case):
    # a coarse form reads the rows at its own width; the operations are the
    # inner products of every query with every row
    width = {EXACT: 4, BF16: 2, FP8: 1}[case["form"]]
    if case["kind"] == "batch":
        dbs, batches = _spec(case)
        return {"bytes": sum(n * d * width for n, d in dbs) + sum(nq * (dbs[i][1] * 4 + k * 8) for i, nq, k in batches),
                "flops": sum(2 * nq * dbs[i][0] * dbs[i][1] for i, nq, _ in batches)}
    q = sum(_sizes(case)) if case["kind"] == "serve" else case["q"]
    n, d, k = case["n"], case["d"], case["k"]
    return {"bytes": n * d * width + q * (d * 4 + k * 8), "flops": 2 * q * n * d}


# ---------------------------------------------------------------- 64 bits
def _nearest(rows, queries, k):
    """Sorted squared distances of the k nearest rows of every query (FP64).
    The k smallest lie in the k blocks of 64 rows with the smallest minima."""
    n = rows.shape[0]
    k = min(k, n)
    x = rows.double()
    xn = (x * x).sum(1)
    blocks = (n + 63) // 64
    out = torch.empty((queries.shape[0], k), dtype=torch.float64, device=rows.device)
    step = max(1, min(queries.shape[0], 1_500_000_000 // n))
    d2 = torch.full((step, blocks * 64), math.inf, dtype=torch.float64, device=rows.device)
    for a in range(0, queries.shape[0], step):
        q = queries[a:a + step].double()
        t = d2[:q.shape[0]]
        torch.addmm(xn[None, :], q, x.t(), alpha=-2.0, out=t[:, :n]) if n == t.shape[1] else \
            t[:, :n].copy_(torch.addmm(xn[None, :], q, x.t(), alpha=-2.0))
        t = t.view(q.shape[0], blocks, 64)
        near = t.amin(2).topk(min(k, blocks), dim=1, largest=False).indices
        near = t.gather(1, near[:, :, None].expand(-1, -1, 64)).flatten(1)
        near = near.topk(k, dim=1, largest=False).values + (q * q).sum(1)[:, None]
        out[a:a + step] = near.clamp_(min=0.0).sort(1).values
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        rows, queries = _batch_inputs(case, seed)
        dist = torch.cat([_nearest(rows[db], q, k).flatten() for (db, _, k), q in zip(_spec(case)[1], queries)])
        return {"distances": dist, "indices": None}
    q = sum(_sizes(case)) if case["kind"] == "serve" else case["q"]
    rows, queries = _table(case, seed, q)
    dist = _nearest(rows, queries, case["k"])
    return {"distances": dist.flatten() if case["kind"] == "serve" else dist, "indices": None}
