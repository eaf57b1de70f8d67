"""Workers prepared by several threads at once hold scratch of their own: all of
them stay alive and are run after every thread has prepared its share, on scratch
that earlier workers of any thread gave back. Calls run one at a time (an index
is used by one stream at a time). Bit-exact against the oracle."""
import threading

import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N_ADS = 70_001
NW = (N_ADS + 31) // 32
THREADS, ROUNDS = 4, 4


def test_workers_of_all_threads_keep_their_scratch(dev):
    import torch
    spec = W.ListsSpec(n_terms=5003, n_ads=N_ADS, nnz=200_000, zipf_s=1.1, max_len=20_000, seed=101)
    off, ads = W.gen_lists(spec)
    qoff, qt = W.gen_queries(W.QueriesSpec(300, "lognormal", 12.0, 1.5, 1, 600, seed=102), np.diff(off).astype(np.uint32))
    qs = [qt[qoff[i]:qoff[i + 1]].copy() for i in range(300)]
    want = [O.ids_to_bitmap(O.kway_union(off, ads, q), NW) for q in qs]
    host = np.zeros((300, (spec.n_terms + 127) // 128 * 16), np.uint8)
    for i, q in enumerate(qs):
        b = O.term_bitmap_bytes(q, spec.n_terms, pad_to=1)
        host[i, :b.size] = b
    ix = Index.from_csr(off, ads, spec.n_terms, N_ADS)
    one_at_a_time, ready = threading.Lock(), threading.Barrier(THREADS)
    bad = []

    def check(w, kind, q0, n):
        out = torch.zeros((n, NW), dtype=torch.int32, device="cuda")
        if kind == "one":
            ab.ListUnion_sparse(w, out)
        elif kind == "keys":
            qidx = np.repeat(np.arange(n, dtype=np.int32), [qs[q0 + i].size for i in range(n)])
            ab.BatchListUnion_sparse(w, out, torch.from_numpy(qidx).cuda(), NW * 4)
        else:
            ab.BatchListUnion_dense(w, None, out, NW)
        got = out.cpu().numpy().view(np.uint32)
        for i in range(n):
            assert np.array_equal(got[i], want[q0 + i]), (kind, q0, i)

    def work(k):
        try:
            for r in range(ROUNDS):
                q0, n = 10 * k + r, 3 + 37 * ((k + r) % 3)
                mine = [(ix.Prepare(qs[q0]), "one", q0, 1), (ix.Prepare(np.concatenate(qs[q0:q0 + n])), "keys", q0, n),
                        (ix.PrepareBatch(n, host.shape[1], host[q0:q0 + n]), "dense", q0, n)]
                ready.wait(60)
                for m in mine:
                    with one_at_a_time:
                        check(*m)
                ready.wait(60)
                for m in mine:
                    m[0].free()
        except Exception as e:  # reported by the main thread
            bad.append(e)
            ready.abort()

    th = [threading.Thread(target=work, args=(k,)) for k in range(THREADS)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad, bad
