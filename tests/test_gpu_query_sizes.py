"""abf_query at the sizes where its terms change their way to the device (with
the plan kernel's arguments in one of two sizes, or by an upload), several calls
in a row without waiting, on every path, against the oracle."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 111, 112, 113, 799, 800, 801, 1100, 3]


@pytest.mark.parametrize("path", [ab.PATH_AUTO, ab.PATH_PROBE, ab.PATH_UNION, ab.PATH_HYBRID, ab.PATH_TILE])
def test_terms_by_size(dev, path):
    import torch
    spec = W.ListsSpec(n_terms=4001, n_ads=70_001, nnz=200_000, zipf_s=1.1, max_len=20_000, seed=41)
    off, ads = W.gen_lists(spec)
    ix = Index.from_csr(off, ads, spec.n_terms, spec.n_ads)
    n_words = (spec.n_ads + 31) // 32
    rng = np.random.default_rng(7)
    qs = [rng.choice(spec.n_terms + 5, n, replace=False).astype(np.uint32) for n in SIZES]  # a few past the domain
    stride = (n_words + 3) // 4 * 4
    bm = torch.full((len(qs), stride), -1, dtype=torch.int32, device="cuda")
    ids = torch.full((len(qs), spec.n_ads), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((len(qs),), -1, dtype=torch.int64, device="cuda")
    for _ in range(2):
        for i, q in enumerate(qs):  # each call's terms may be overwritten as soon as it returns
            t = q.copy()
            ix.query(t, bm[i], path=path, d_ids=ids[i], d_count=cnt[i:i + 1])
            t[:] = 0
    torch.cuda.synchronize()
    for i, q in enumerate(qs):
        e = O.kway_union(off, ads, q[q < spec.n_terms])
        assert cnt[i].item() == e.size, SIZES[i]
        assert np.array_equal(ids[i, :e.size].cpu().numpy().view(np.uint32), e), SIZES[i]
        assert np.array_equal(bm[i, :n_words].cpu().numpy().view(np.uint32), O.ids_to_bitmap(e, n_words)), SIZES[i]
