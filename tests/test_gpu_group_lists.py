"""Lists of the dense group kernel: every length modulo its steps of 16, 8, 4, 2
and 1 rows, lists that fit in shared memory and that do not, both tile widths,
one and several windows, against numpy."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_dense", [1, 17, 400, 700])
@pytest.mark.parametrize("n_q", [32, 300, 2049])
@pytest.mark.parametrize("gw", [64, 32])
def test_group_lists(dev, n_dense, n_q, gw):
    import torch
    n_ads, n_terms = 9_001, n_dense + 5
    rng = np.random.default_rng(n_dense)
    rows = np.zeros((n_terms, n_ads), bool)
    for t in range(n_terms):  # lengths fall with the term, so dense bitmap t is term t's
        n = 1000 - t if t < n_dense else 3
        rows[t, rng.choice(n_ads, n, replace=False)] = True
    off = np.concatenate([[0], np.cumsum(rows.sum(1))]).astype(np.uint64)
    ix = Index.from_csr(off, np.flatnonzero(rows.ravel()).astype(np.uint64) % n_ads, n_terms, n_ads, dense_div=40)
    assert ix.stats()["n_dense_lists"] == n_dense
    ix.set_tuning(group_tile_words=gw)
    qs = []
    for i in range(n_q):
        if i < 64:  # every length from none to 63 (or all the lists), the sparsest ones: no early exit
            q = list(range(max(0, n_dense - i), n_dense)) + ([n_terms - 1] if i % 3 else [])
        else:
            q = rng.choice(n_terms, int(rng.integers(0, min(n_terms, 60))), replace=False).tolist()
        qs.append(np.array(q, np.uint32))
    terms = np.concatenate(qs + [np.zeros(1, np.uint32)])
    qoff = np.concatenate([[0], np.cumsum([q.size for q in qs])]).astype(np.uint64)
    n_words = (n_ads + 31) // 32
    stride = (n_words + 3) // 4 * 4
    bm = torch.full((n_q, stride), -1, dtype=torch.int32, device="cuda")
    ws = ix.workspace(n_q, terms.size)
    ix.batch_run(ws, torch.from_numpy(terms.view(np.int32)).cuda(), torch.from_numpy(qoff.view(np.int64)).cuda(), n_q, bm,
                 stride, path=ab.PATH_UNION)
    ws.check()
    got = np.unpackbits(bm.cpu().numpy().view(np.uint8)[:, :n_words * 4], axis=1, bitorder="little")[:, :n_ads]
    for i, q in enumerate(qs):
        q = q[q < n_terms]
        assert np.array_equal(got[i].astype(bool), rows[q].any(0) if q.size else np.zeros(n_ads, bool)), i
