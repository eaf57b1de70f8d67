"""Queries whose offsets leave the workspace's terms (or run backwards) get no
work on any path: an empty bitmap, no ids, an error to read, the path of an
empty query, and neighbours that are answered as ever. The terms lie in a larger
array, so that offsets too large still name allocated memory."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, planner as P, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ABF_ERR_CAPACITY = 8
N_ADS = 70_001


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=3001, n_ads=N_ADS, nnz=300_000, zipf_s=1.1, max_len=20_000, seed=61)
    off, ads = W.gen_lists(spec)
    return dict(off=off, ads=ads, lens=np.diff(off).astype(np.uint32), ix=Index.from_csr(off, ads, spec.n_terms, N_ADS))


def counting_planner():
    """UNION for a query without terms (0 against 1 and 99), HYBRID for one of two terms or more (ln(1 + n) > 1)."""
    p = P.init_params(np.zeros(P.F, np.float32), np.ones(P.F, np.float32), seed=1)
    p[P.OFF["W1"]:] = 0
    p[P.OFF["W1"]] = p[P.OFF["W2"]] = p[P.OFF["W3"] + 64] = 1  # union's output: feature 0, ln(1 + terms)
    p[P.OFF["b3"]:] = [99, 0, 1]
    return p


@pytest.mark.parametrize("n", [3, 40, 2100])  # stream, group, and scan kernels
@pytest.mark.parametrize("what", ["planner", "auto", "union", "hybrid"])
def test_offsets_past_the_terms(env, n, what):
    import torch
    ix = env["ix"]
    qoff, qt = W.gen_queries(W.QueriesSpec(n, "uniform", 0.0, 0.0, 4, 30, seed=62), env["lens"])
    cap = int(qt.size)
    terms = torch.from_numpy(np.resize(qt, 4 * cap + 4096).view(np.int32)).cuda()
    path = {"union": ab.PATH_UNION, "hybrid": ab.PATH_HYBRID}.get(what, ab.PATH_AUTO)
    back, over = qoff.copy(), qoff.copy()
    # only the last query's end is off: another one's would be the next query's
    # beginning and give both the same slots
    back[n] = qoff[n - 1] - 1
    over[n] = 4 * cap
    nw = (N_ADS + 31) // 32
    stride = (nw + 3) // 4 * 4
    ws = ix.workspace(n, cap)
    if what == "planner":
        P.install(ix, counting_planner())
    try:
        for offs, bad in ((back, n - 1), (over, n - 1), (qoff, None)):
            bm = torch.full((n, stride), -1, dtype=torch.int32, device="cuda")
            ids = torch.zeros(n * N_ADS, dtype=torch.int32, device="cuda")
            idoff = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
            ix.batch_run(ws, terms, torch.from_numpy(offs.view(np.int64)).cuda(), n, bm, stride, path=path, d_ids=ids,
                         d_id_offsets=idoff)
            if bad is None:
                ws.check()
            else:
                with pytest.raises(ab.AbfError) as e:
                    ws.check()
                assert e.value.status == ABF_ERR_CAPACITY
            paths = ws.paths(n)
            got, io = bm.cpu().numpy().view(np.uint32), idoff.cpu().numpy()
            host_terms = np.resize(qt, 4 * cap + 4096)
            for i in sorted({0, 1, 2, n // 2, n - 2, n - 1}):
                q = host_terms[:0] if i == bad else host_terms[int(offs[i]):int(offs[i + 1])]
                want = O.kway_union(env["off"], env["ads"], q) if q.size else np.array([], np.uint32)
                assert np.array_equal(got[i, :nw], O.ids_to_bitmap(want, nw)), i
                assert np.array_equal(ids[io[i]:io[i + 1]].cpu().numpy().view(np.uint32), want), i
                if what == "planner":
                    assert paths[i] == (ab.PATH_HYBRID if q.size else ab.PATH_UNION), i
    finally:
        if what == "planner":
            P.uninstall(ix)


@pytest.mark.parametrize("n", [3, 40, 2100])
@pytest.mark.parametrize("path", [ab.PATH_UNION, ab.PATH_HYBRID, ab.PATH_TILE])
def test_queries_over_one_another(env, n, path):
    """A query that ends before it begins gives those after it slots of those before: the batch gets no work, an
    error to read, and the next batch is answered as ever."""
    import torch
    ix = env["ix"]
    qoff, qt = W.gen_queries(W.QueriesSpec(n, "uniform", 0.0, 0.0, 4, 30, seed=63), env["lens"])
    terms = torch.from_numpy(qt.view(np.int32)).cuda()
    nw = (N_ADS + 31) // 32
    stride = (nw + 3) // 4 * 4
    ws = ix.workspace(n, qt.size)
    back = qoff.copy()
    back[n // 2], back[n // 2 + 1] = qoff[n // 2 + 1], qoff[n // 2]
    for offs, good in ((back, False), (qoff, True)):
        bm = torch.full((n, stride), -1, dtype=torch.int32, device="cuda")
        idoff = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")
        ids = torch.zeros(n * 4096 if not good else n * N_ADS, dtype=torch.int32, device="cuda")
        ix.batch_run(ws, terms, torch.from_numpy(offs.view(np.int64)).cuda(), n, bm, stride, path=path, d_ids=ids,
                     d_id_offsets=idoff)
        if not good:
            with pytest.raises(ab.AbfError) as e:
                ws.check()
            assert e.value.status == ABF_ERR_CAPACITY
            assert not bm[:, :nw].any() and not idoff.any()
            continue
        ws.check()
        got = bm.cpu().numpy().view(np.uint32)
        for i in sorted({0, n // 2, n - 1}):
            assert np.array_equal(got[i, :nw], O.ids_to_bitmap(O.kway_union(env["off"], env["ads"], qt[qoff[i]:qoff[i + 1]]), nw)), i
