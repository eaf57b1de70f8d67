"""Bounded waits of the operators' kernels that run out are reported: the
worker's error flag starts clear whatever its scratch held before, keeps the
failure for the check, and the worker goes on answering. Nothing here faults or
hangs: the self-test's waits are on a copy that is never issued and a word that
nothing publishes, and give up after a few thousand polls."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ABF_ERR_TIMEOUT = 7
N_ADS = 70_001
NW = (N_ADS + 31) // 32


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=3001, n_ads=N_ADS, nnz=200_000, zipf_s=1.1, max_len=20_000, seed=81)
    off, ads = W.gen_lists(spec)
    qoff, qt = W.gen_queries(W.QueriesSpec(300, "lognormal", 12.0, 1.5, 1, 600, seed=82), np.diff(off).astype(np.uint32))
    qs = [qt[qoff[i]:qoff[i + 1]].copy() for i in range(300)]
    host = np.zeros((300, (spec.n_terms + 127) // 128 * 16), np.uint8)
    for i, q in enumerate(qs):
        b = O.term_bitmap_bytes(q, spec.n_terms, pad_to=1)
        host[i, :b.size] = b
    ix = Index.from_csr(off, ads, spec.n_terms, N_ADS)
    return dict(ix=ix, qs=qs, host=host, want=np.stack([O.ids_to_bitmap(O.kway_union(off, ads, q), NW) for q in qs]))


@pytest.mark.parametrize("n", [1, 40, 300])  # 300: two windows of query bitmaps
@pytest.mark.parametrize("kind", ["device", "host", "keys"])
def test_worker_reports_waits_that_ran_out(env, kind, n):
    import torch
    ix, host = env["ix"], env["host"][:n]
    up = torch.from_numpy(host).cuda()
    qidx = torch.from_numpy(np.repeat(np.arange(n, dtype=np.int32), [q.size for q in env["qs"][:n]])).cuda()

    def prepare():
        if kind == "device":
            return ix.PrepareBatchDevice(n, host.shape[1], up)
        return ix.PrepareBatch(n, host.shape[1], host) if kind == "host" else ix.Prepare(np.concatenate(env["qs"][:n]))

    def run(w):
        out = torch.zeros((n, NW), dtype=torch.int32, device="cuda")
        if kind == "keys":
            ab.BatchListUnion_sparse(w, out, qidx, NW * 4)
        else:
            ab.BatchListUnion_dense(w, None, out, NW)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), env["want"][:n])

    w = prepare()
    w.check()  # before any call
    for _ in range(2):
        w.selftest_waits(1 << 12)
        with pytest.raises(ab.AbfError) as e:
            w.check()
        assert e.value.status == ABF_ERR_TIMEOUT
        assert "code 3" in str(e.value)  # the mbarrier wait (2) and the look-back wait (1)
        w.check()  # read and cleared
        run(w)
        w.check()
    # the next worker gets the same scratch, with the flag of the one before set
    w.selftest_waits(1 << 12)
    w.free()
    w = prepare()
    w.check()
    run(w)
    w.check()
