"""The bitmap-probe scan at the edges of its chunks and steps of 32 blocks.
Bit-exact against the oracle."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N_ADS = 60_013


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=701, n_ads=N_ADS, nnz=150_000, zipf_s=1.1, max_len=30_000, seed=61)
    off, ads = W.gen_lists(spec)
    qoff, qt = W.gen_queries(W.QueriesSpec(70, "lognormal", 8.0, 1.2, 1, 300, seed=62), np.diff(off).astype(np.uint32))
    return dict(spec=spec, off=off, ads=ads, qoff=qoff, qt=qt)


@pytest.mark.parametrize("chunk", [128, 256, 384, 4096])
@pytest.mark.parametrize("n_q", [1, 32, 33, 70])
def test_probe_chunks(env, chunk, n_q):
    import torch
    ix = Index.from_csr(env["off"], env["ads"], env["spec"].n_terms, N_ADS)
    ix.set_tuning(probe_chunk_blocks=chunk, probe_cap=128)
    qoff, qt = env["qoff"][:n_q + 1], env["qt"][:int(env["qoff"][n_q])]
    nw = (N_ADS + 31) // 32
    stride = (nw + 3) // 4 * 4
    bm = torch.zeros((n_q, stride), dtype=torch.int32, device="cuda")
    d_off = torch.from_numpy(np.ascontiguousarray(qoff, np.uint64).view(np.int64)).cuda()
    d_qt = torch.from_numpy(np.ascontiguousarray(qt, np.uint32).view(np.int32)).cuda()
    ix.batch_run(ix.workspace(n_q, qt.size), d_qt, d_off, n_q, bm, stride, path=ab.PATH_PROBE)
    got = bm.cpu().numpy().view(np.uint32)
    for i in range(n_q):
        want = O.ids_to_bitmap(O.kway_union(env["off"], env["ads"], qt[int(qoff[i]):int(qoff[i + 1])]), nw)
        assert np.array_equal(got[i, :nw], want), i
