"""Batches on PATH_TILE around the size from which the bin kernel takes the plain
lists (more than 32 tiles of 2^19 ads in all), with lists of every kind and
without scattering. Bit-exact against the oracle."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[70_001, 3 * (1 << 19) + 5])  # 1 and 4 tiles
def env(dev, request):
    n_ads = request.param
    spec = W.ListsSpec(n_terms=4001, n_ads=n_ads, nnz=900_000, zipf_s=1.1, max_len=n_ads // 4, seed=111)
    off, ads = W.gen_lists(spec)
    lens = np.diff(off).astype(np.uint32)
    ix = Index.from_csr(off, ads, spec.n_terms, n_ads)
    flags = ix.list_flags()
    assert (flags & 1).any() and ((flags & 1 == 0) & (lens >= 256)).any() and (lens < 256).any()
    qoff, qt = W.gen_queries(W.QueriesSpec(40, "lognormal", 12.0, 1.5, 1, 600, seed=112), lens)
    return dict(n_ads=n_ads, ix=ix, qoff=qoff, qt=qt,
                want=[O.kway_union(off, ads, qt[qoff[i]:qoff[i + 1]]) for i in range(40)])


@pytest.mark.parametrize("n", [1, 2, 8, 9, 31, 32, 33, 40])
@pytest.mark.parametrize("group", [0, 32])
def test_tile_batches(env, n, group):
    import torch
    ix, n_ads = env["ix"], env["n_ads"]
    ix.set_tuning(group_min_queries=group)
    nw = (n_ads + 31) // 32
    for stride in ((nw + 3) // 4 * 4, nw | 1):  # the second: rows that are not 16-byte aligned
        ws = ix.workspace(n, int(env["qoff"][n]))
        bm = torch.full((n, stride), -1, dtype=torch.int32, device="cuda")
        ids = torch.zeros(sum(env["want"][i].size for i in range(n)) + 1, dtype=torch.int32, device="cuda")
        idoff = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        ix.batch_run(ws, torch.from_numpy(env["qt"].view(np.int32)).cuda(),
                     torch.from_numpy(env["qoff"].view(np.int64)).cuda(), n, bm, stride, path=ab.PATH_TILE, d_ids=ids,
                     d_id_offsets=idoff)
        ws.check()
        got, got_ids, o = bm.cpu().numpy().view(np.uint32), ids.cpu().numpy().view(np.uint32), idoff.cpu().numpy()
        for i in range(n):
            assert np.array_equal(got[i, :nw], O.ids_to_bitmap(env["want"][i], nw)), i
            assert np.array_equal(got_ids[o[i]:o[i + 1]], env["want"][i]), i
