"""The work a user of the library has it do, as measurable cases.

An index is built once and then answers queries for a long time, so here it is
part of what a program has in hand: it is built once per shape (from the shape
alone) and kept, as a service would keep it. The queries, the bitmaps to
compact and the training samples are the inputs; they come from the seed.

The shapes are the repository's own workloads (adabool_b200/workload.py): c0
(65,536 terms x 2^20 ads, 8M postings), c1 (2^20 terms x 2^24 ads, 500M
postings) and c1 at a quarter scale, with an odd number of ads in places.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import adabool_b200 as ab
from adabool_b200 import planner as P
from adabool_b200 import workload as W
from adabool_b200._native import check, lib, ptr
from adabool_b200.executor import GraphBatchExecutor

PATHS = {"auto": ab.PATH_AUTO, "union": ab.PATH_UNION, "hybrid": ab.PATH_HYBRID, "tile": ab.PATH_TILE,
         "probe": ab.PATH_PROBE}

C0 = dict(n_terms=65536, n_ads=1 << 20, nnz=8_000_000, zipf=1.1, max_len=200_000)
# the full-size service: dense bitmaps for lists of n_ads/256 postings, the
# tuner's settings for that index, a trained planner installed
C1 = dict(n_terms=1 << 20, n_ads=1 << 24, nnz=500_000_000, zipf=1.05, max_len=5_000_000, service=True)
# a quarter of it, with the library's defaults and an ad count that fills no word
MID = dict(n_terms=1 << 18, n_ads=(1 << 22) - 3, nnz=125_000_000, zipf=1.05, max_len=1_250_000)


def listed():
    return [
        # one small request: latency of a single call, terms in, bitmap and ids out
        dict(C0, name="query_small", op="query", queries=1, kind="uniform", lo=4, hi=64, path="auto", ids=True),
        # one request against the full-size index, path by the installed planner
        dict(C1, name="query_full", op="query", queries=1, kind="lognormal", median=40, sigma=1.5, lo=1, hi=5000,
             path="auto", ids=True),
        # an offline batch on the small index
        dict(C0, name="batch_small", op="batch", queries=256, kind="uniform", lo=4, hi=64, path="auto", ids=True),
        # what the serving loop launches at a time under moderate load
        dict(C1, name="serve_full", op="batch", queries=7, kind="lognormal", median=40, sigma=2.0, lo=1, hi=20000,
             path="auto", ids=True),
        # the throughput workload: bitmaps and sorted ids of a large batch
        dict(C1, name="batch_full", op="batch", queries=512, kind="lognormal", median=40, sigma=1.5, lo=1, hi=5000,
             path="union", ids=True),
        # uneven queries through one CUDA-graph launch, bitmaps only
        dict(C1, name="graph_full", op="graph", queries=2048, kind="lognormal", median=40, sigma=2.0, lo=1, hi=20000,
             path="union", ids=False),
        # long lists merged per tile, short ones scattered; odd sizes throughout
        dict(MID, name="hybrid_mid", op="batch", queries=61, kind="lognormal", median=40, sigma=1.5, lo=1, hi=5000,
             path="hybrid", ids=True),
        # the reference-shaped operators: batched bitmap-probe at the reference's own batch limit ...
        dict(MID, name="probe_mid", op="probe", queries=32, kind="lognormal", median=40, sigma=1.5, lo=1, hi=5000),
        # ... list-union of one prepared query ...
        dict(MID, name="union_mid", op="union", queries=1, kind="lognormal", median=40, sigma=1.5, lo=1, hi=5000),
        # ... and of a flattened batch with a query index per key
        dict(MID, name="union_keys_mid", op="union_keys", queries=32, kind="lognormal", median=40, sigma=1.5, lo=1,
             hi=5000),
        # compaction alone: bitmaps of every density to sorted ids
        dict(MID, name="collect_mid", op="collect", queries=64),
        # one optimiser step of the planner's training at the trainer's batch size
        dict(name="train_step", op="train", n=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["query", "query", "batch", "batch", "batch", "batch", "graph", "probe", "union", "union_keys",
                     "collect", "train"])
    if op == "train":
        return dict(op="train", n=_log(rng, 500, 200_000))
    n_ads = _log(rng, 1 << 18, 1 << 24)
    per_ad = rng.uniform(7.0, 30.0)
    case = dict(op=op, n_terms=_log(rng, n_ads // 32 + 1, n_ads // 12), n_ads=n_ads, nnz=int(per_ad * n_ads),
                zipf=round(rng.uniform(1.05, 1.1), 3), max_len=int(n_ads * rng.uniform(0.18, 0.3)),
                service=rng.random() < 0.3)
    room = (512 << 24) // n_ads
    if op in ("query", "union"):
        n = 1
    elif op in ("probe", "union_keys"):
        n = rng.randint(2, 32)
    elif op == "collect":
        n = _log(rng, 1, min(room // 4, 512))
    elif op == "graph":
        n = _log(rng, 64, min(room, 2048))
    else:
        n = _log(rng, 1, min(room, 1024))
    case.update(queries=n)
    if op == "collect":
        return case
    if rng.random() < 0.3:
        case.update(kind="uniform", lo=4, hi=64)
    else:
        case.update(kind="lognormal", median=40, sigma=rng.choice([1.5, 2.0]), lo=1, hi=5000)
    if op in ("query", "batch", "graph"):
        case.update(path=rng.choice(["auto", "auto", "union", "union", "hybrid"]), ids=op != "graph" and rng.random() < 0.8)
    return case


# ---------------------------------------------------------------------------
def _planner_params():
    """Parameters as a trained planner has them on these workloads: list-union is predicted cheapest for nearly
    every query, the bitmap-probe scan dearest."""
    p = P.init_params(np.full(P.F, 4.0, np.float32), np.full(P.F, 4.0, np.float32), seed=3)
    p[P.OFF["W3"]:P.OFF["b3"]] *= 0.05
    p[P.OFF["b3"]:] = [7.0, 4.0, 4.3]
    return p


@functools.lru_cache(maxsize=2)
def _index(n_terms, n_ads, nnz, zipf, max_len, service):
    off, ads = W.gen_lists(W.ListsSpec(n_terms, n_ads, nnz, zipf, max_len, seed=21))
    ix = ab.Index.from_csr(off, ads, n_terms, n_ads, dense_div=256 if service else 0)
    if service:
        ix.set_tuning(tile_words=256, warps_per_tile=8, heavy_min_len=max(128, n_ads // 128),
                      scatter_blocks_per_warp=8, ctas_per_sm=8, group_min_queries=32)
        P.install(ix, _planner_params())
    return ix, ix.list_lengths()


def _the_index(case):
    return _index(case["n_terms"], case["n_ads"], case["nnz"], case["zipf"], case["max_len"],
                  bool(case.get("service")))


def _queries(case, lens, seed):
    return W.gen_queries(W.QueriesSpec(case["queries"], case["kind"], float(case.get("median", 40)),
                                       float(case.get("sigma", 1.5)), case["lo"], min(case["hi"], case["n_terms"]),
                                       seed=1000 + seed), lens)


def _term_bitmaps(off, terms, n_terms):
    length = (n_terms + 127) // 128 * 16
    bm = np.zeros((off.size - 1, length * 8), np.uint8)
    bm[np.repeat(np.arange(off.size - 1), np.diff(off.astype(np.int64))), terms] = 1
    return length, torch.from_numpy(np.packbits(bm, axis=1, bitorder="little")).cuda()


def _random_bitmaps(n, n_words, stride, seed):
    """Bitmaps from nearly empty to full, each of one density, as unions of uniformly drawn lists are."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def words():
        return torch.randint(-(1 << 31), 1 << 31, (n_words,), generator=g, device="cuda",
                             dtype=torch.int64).to(torch.int32)

    bm = torch.zeros((n, stride), dtype=torch.int32, device="cuda")
    kinds = torch.randint(0, 13, (n,), generator=torch.Generator().manual_seed(seed)).tolist()
    for i, k in enumerate(kinds):
        if k == 12:  # every ad matches
            bm[i, :n_words] = -1
            continue
        w = words()
        for _ in range(k % 6):
            w = w & words() if k < 6 else w | words()
        bm[i, :n_words] = w
    return bm


MLP = [(64, 16), (64, 64), (3, 64)]


def _train_state(n, seed):
    """A batch and the optimiser's state in mid-training (parameter layout of include/adabool.h)."""
    r = np.random.default_rng(seed)
    x = r.normal(size=(n, 16))
    parts = [np.zeros(16), np.ones(16)]
    for rows, cols in MLP:
        parts += [r.normal(0, math.sqrt(2.0 / cols), rows * cols), r.normal(0, 0.1, rows)]
    p = np.concatenate(parts)
    t = 4.0 + x[:, :3] + r.normal(0, 0.3, (n, 3))
    mask = (r.random((n, 3)) < 0.95)
    m = r.normal(0, 0.01, p.size)
    v = r.uniform(0.001, 0.01, p.size)
    return [np.ascontiguousarray(a, np.float32) for a in (p, x, t, mask, m, v)]


def prepare(case, seed):
    op = case["op"]
    if op == "train":
        p, x, t, mask, m, v = (torch.from_numpy(a).cuda() for a in _train_state(case["n"], seed))
        return dict(op=op, n=case["n"], p=p, x=x, t=t, mask=mask, m=m, v=v, g=torch.zeros_like(p),
                    loss=torch.zeros(2, device="cuda"), step=1000)
    ix, lens = _the_index(case)
    n = case["queries"]
    stride = (ix.n_words + 3) // 4 * 4
    s = dict(op=op, ix=ix, n=n, stride=stride)
    if op == "collect":
        s.update(bm=_random_bitmaps(n, ix.n_words, stride, seed), ws=ix.workspace(n, 1),
                 ids=torch.zeros(n * ix.n_ads, dtype=torch.int32, device="cuda"),
                 off=torch.zeros(n + 1, dtype=torch.int64, device="cuda"))
        return s
    off, terms = _queries(case, lens, seed)
    s.update(path=PATHS[case["path"]] if "path" in case else None)
    if op == "union":
        s.update(worker=ix.Prepare(terms), bm=torch.zeros(stride, dtype=torch.int32, device="cuda"))
        return s
    if op in ("probe", "union_keys"):
        s.update(bm=torch.zeros((n, stride), dtype=torch.int32, device="cuda"))
        if op == "probe":
            length, d = _term_bitmaps(off, terms, ix.n_terms)
            s.update(worker=ix.PrepareBatchDevice(n, length, d))
        else:
            qidx = np.repeat(np.arange(n, dtype=np.int32), np.diff(off.astype(np.int64)))
            s.update(worker=ix.Prepare(terms), qidx=torch.from_numpy(qidx).cuda())
        return s
    room = n * ix.n_ads  # every ad could match
    if op == "query":
        s.update(terms=terms, bm=torch.zeros(stride, dtype=torch.int32, device="cuda"), ids=None, count=None)
        if case["ids"]:
            s.update(ids=torch.zeros(room, dtype=torch.int32, device="cuda"),
                     count=torch.zeros(1, dtype=torch.int64, device="cuda"))
        return s
    s.update(terms=torch.from_numpy(terms.view(np.int32)).cuda(), off=torch.from_numpy(off.view(np.int64)).cuda())
    if op == "graph":
        s.update(ex=GraphBatchExecutor(ix, n, terms.size, path=s["path"]).capture())
        return s
    s.update(ws=ix.workspace(n, terms.size), bm=torch.zeros((n, stride), dtype=torch.int32, device="cuda"), ids=None,
             idoff=None)
    if case["ids"]:
        s.update(ids=torch.zeros(room, dtype=torch.int32, device="cuda"),
                 idoff=torch.zeros(n + 1, dtype=torch.int64, device="cuda"))
    return s


def run(s):
    op = s["op"]
    if op == "train":
        s["step"] += 1
        check(lib().abf_mlp_grad(ptr(s["p"]), ptr(s["x"]), ptr(s["t"]), ptr(s["mask"]), s["n"], ptr(s["g"]),
                                 ptr(s["loss"]), None))
        check(lib().abf_mlp_adam(ptr(s["p"]), ptr(s["g"]), ptr(s["m"]), ptr(s["v"]), s["step"], 2e-3, 0.9, 0.999,
                                 1e-8, None))
        return dict(grad=s["g"], loss=s["loss"], params=s["p"], m=s["m"], v=s["v"])
    ix = s["ix"]
    if op == "query":
        ix.query(s["terms"], s["bm"], path=s["path"], d_ids=s["ids"], d_count=s["count"])
        return dict(bitmap=s["bm"], ids=s["ids"], count=s["count"])
    if op == "batch":
        ix.batch_run(s["ws"], s["terms"], s["off"], s["n"], s["bm"], s["stride"], path=s["path"], d_ids=s["ids"],
                     d_id_offsets=s["idoff"])
        return dict(bitmaps=s["bm"], ids=s["ids"], offsets=s["idoff"])
    if op == "graph":
        ex, here = s["ex"], torch.cuda.current_stream()
        ex.stream.wait_stream(here)
        ex.set_batch_device(s["off"], s["terms"], s["n"])
        ex.replay()
        here.wait_stream(ex.stream)
        return dict(bitmaps=ex.bitmaps)
    if op == "collect":
        ab.BatchCollectIds(ix, s["ws"], s["bm"], s["stride"], s["n"], s["ids"], s["off"])
        return dict(ids=s["ids"], offsets=s["off"])
    s["bm"].zero_()  # the operators OR into the caller's bitmap
    if op == "union":
        ab.ListUnion_sparse(s["worker"], s["bm"])
    elif op == "probe":
        ab.BatchListUnion_dense(s["worker"], None, s["bm"], s["stride"])
    else:
        ab.BatchListUnion_sparse(s["worker"], s["bm"], s["qidx"], s["stride"] * 4)
    return dict(bitmaps=s["bm"])


# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _target_lengths(n_terms, n_ads, nnz, zipf, max_len):
    return W.target_lengths(W.ListsSpec(n_terms, n_ads, nnz, zipf, max_len, seed=21))


def work(case):
    """Bytes of one pass: every list that a query names read once in the smaller of its two forms (bitmap, or gaps
    at about their entropy), every output written once; ids by the expected size of the union."""
    if case["op"] == "train":
        n, params = case["n"], 32 + sum(r * c + r for r, c in MLP)
        # forward, and two products of the same size backward
        return {"bytes": 4.0 * (n * (16 + 3 + 3) + 8 * params), "flops": 6.0 * n * sum(r * c for r, c in MLP)}
    n, n_ads = case["queries"], case["n_ads"]
    if case["op"] == "collect":
        # the densities of _random_bitmaps: half each for k = 0 and 6, 2^-(k+1) or its complement, one kind full
        mean = (sum(2.0 ** -(k + 1) for k in range(6)) + sum(1 - 2.0 ** -(k + 1) for k in range(6)) + 1.0) / 13
        return {"bytes": n * (n_ads / 8 + 4 * mean * n_ads), "flops": 0.0}
    lens = _target_lengths(case["n_terms"], n_ads, case["nnz"], case["zipf"], case["max_len"])
    off, terms = _queries(case, lens, 0)
    used = lens[np.unique(terms)].astype(np.float64)
    gaps = used * (np.log2(n_ads / used) + 1.5) / 8
    total = float(np.minimum(gaps, n_ads / 8).sum()) + n * n_ads / 8 + 4.0 * terms.size
    if case["op"] == "probe":
        total += n * case["n_terms"] / 8
    if case.get("ids"):
        log_none = np.add.reduceat(np.log1p(-lens[terms].astype(np.float64) / n_ads), off[:-1].astype(np.int64))
        total += 4.0 * n_ads * float((1 - np.exp(log_none)).sum())
    return {"bytes": total, "flops": 0.0}


def exact(case, seed):
    """The training step in 64 bits; every other output is whole numbers."""
    if case["op"] != "train":
        return None
    p, x, t, mask, m, v = (torch.from_numpy(a).cuda().double() for a in _train_state(case["n"], seed))
    p0 = p.clone()
    p.requires_grad_(True)
    at, h = 32, x
    for i, (rows, cols) in enumerate(MLP):
        w, b = p[at:at + rows * cols].view(rows, cols), p[at + rows * cols:at + rows * cols + rows]
        at += rows * cols + rows
        h = h @ w.T + b
        h = torch.relu(h) if i < 2 else h
    loss = (mask * (h - t) ** 2).sum() / mask.sum()
    loss.backward()
    g, step = p.grad, 1001
    lr, b1, b2, eps = (float(np.float32(c)) for c in (2e-3, 0.9, 0.999, 1e-8))
    m1, v1 = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
    new = p0 - lr * (m1 / (1 - b1 ** step)) / (torch.sqrt(v1 / (1 - b2 ** step)) + eps)
    at = torch.arange(p.numel(), device="cuda") < 32  # the standardisation entries take no step
    return dict(grad=g, loss=torch.stack([loss.detach(), mask.sum()]), params=torch.where(at, p0, new),
                m=torch.where(at, m, m1), v=torch.where(at, v, v1))
