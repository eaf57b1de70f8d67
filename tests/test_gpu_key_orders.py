"""Keyed list-union with the keys' bitmap indices in every order: sorted (a run
per query), in no order (a key per run), all the same, and runs of lengths around
the eight below which keys past the first 256 runs are taken in chunks; key
counts around one and several planning steps; with the dense bitmaps merged by
the group kernel and scattered. Bit-exact against the oracle."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N_ADS = 70_001
NW = (N_ADS + 31) // 32
STRIDE = NW + 1


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=5003, n_ads=N_ADS, nnz=400_000, zipf_s=1.1, max_len=30_000, seed=121)
    off, ads = W.gen_lists(spec)
    lens = np.diff(off).astype(np.int64)
    ix = Index.from_csr(off, ads, spec.n_terms, N_ADS)
    ix.profile(True)
    lists = np.zeros((spec.n_terms + 1, NW), np.uint32)  # the last row: terms that are none
    for t in range(spec.n_terms):
        lists[t] = O.ids_to_bitmap(ads[off[t]:off[t + 1]], NW)
    return dict(ix=ix, lists=lists, n_terms=spec.n_terms, long=np.flatnonzero(lens * 128 >= N_ADS), lens=lens)


def orders(n, rng):
    yield "sorted", np.sort(rng.integers(0, 40, n))
    yield "mixed", rng.integers(0, 40, n)
    yield "one", np.full(n, 7)
    for run in (7, 8, 9):  # whole runs of this length; the index changes from each to the next
        yield f"runs of {run}", np.arange(n) // run * 11 % 40


@pytest.mark.parametrize("n", [1, 255, 257, 1024, 2048, 2049, 3073, 9001])
@pytest.mark.parametrize("keys", ["any", "long"])
def test_key_orders(env, n, keys):
    import torch
    ix, rng = env["ix"], np.random.default_rng(n)
    k = rng.choice(env["long"], n) if keys == "long" else rng.integers(0, env["n_terms"] + 3, n)
    k = k.astype(np.uint32)
    w = ix.Prepare(k)
    row = np.minimum(k, env["n_terms"])
    postings = int(env["lens"][k].sum()) if keys == "long" else 0
    grouped = postings >= env["long"].size * N_ADS // 64 + (1 << 23)
    assert keys == "any" or grouped or n < 9001
    for name, qidx in orders(n, rng):
        qidx = qidx.astype(np.int32)
        want = np.zeros((40, NW), np.uint32)
        for q in range(40):
            want[q] = np.bitwise_or.reduce(env["lists"][np.unique(row[qidx == q])], axis=0, initial=0)
        d = torch.from_numpy(qidx).cuda()
        for _ in range(2):
            out = torch.zeros((40, STRIDE), dtype=torch.int32, device="cuda")
            ix.profile_read()
            ab.BatchListUnion_sparse(w, out, d, STRIDE * 4)
            ran = ix.profile_read()
            got = out.cpu().numpy().view(np.uint32)
            assert np.array_equal(got[:, :NW], want), name
            assert not got[:, NW:].any(), name
            if keys == "long":
                assert ("dense_group" in ran) == grouped, (name, ran)
    w.check()
