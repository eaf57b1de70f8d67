"""The binned list-union (bin_kernel) against the oracle, at the edges of its
16,384-word tiles, of its length and block thresholds, of its marks (64- and
32-word tiles), with lists whose gaps need more than 16 bits, with queries cut
into parts, and against the same batch without it (group kernel off)."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILE = 16384 * 32


def build(n_ads, seed=3):
    """Lists of every kind over n_ads: dense, mid, short, one with a huge gap per block, runs, tile-edge ids."""
    rng = np.random.default_rng(seed)
    lists = []
    for k in range(400):
        n = int(np.exp(rng.uniform(np.log(20), np.log(max(n_ads // 150, 40)))))
        lists.append(rng.choice(n_ads, size=min(n, n_ads), replace=False))
    for k in range(6):
        lists.append(rng.choice(n_ads, size=n_ads // 20, replace=False))  # dense bitmaps
    for k in range(8):  # 100 ids at the start, then one gap over most of the domain in every block
        a = np.concatenate([np.arange(k, k + 90), rng.choice(n_ads, size=600, replace=False)])
        lists.append(a)
    lists.append(np.arange(min(5000, n_ads)))  # a run: 0-bit gaps
    lists.append(np.arange(0, n_ads, max(1, n_ads // 4000)))
    edges = [x for e in range(0, n_ads + 1, TILE) for x in (e - 1, e, e + 1)] + [n_ads - 1]
    lists.append(np.array([x for x in edges if 0 <= x < n_ads]))
    lists = [np.unique(a).astype(np.uint32) for a in lists]
    off = np.concatenate([[0], np.cumsum([a.size for a in lists])]).astype(np.uint64)
    return off, np.concatenate(lists)


def queries(n_terms, n, rng):
    qs = [rng.choice(n_terms, size=int(rng.integers(1, 60)), replace=False).astype(np.uint32) for _ in range(n)]
    qs[0] = np.arange(n_terms, dtype=np.uint32)  # every list: many parts, mostly saturated
    qs[1] = np.zeros(0, np.uint32)
    qs[2] = np.tile(np.arange(0, 400, 7, dtype=np.uint32), 3)  # repeated terms
    qs[3] = np.concatenate([np.arange(60, dtype=np.uint32), [n_terms, 0xFFFFFFFF]]).astype(np.uint32)
    qs[4] = np.arange(200, 414, dtype=np.uint32)
    return qs


@pytest.mark.parametrize("n_ads", [TILE - 31, TILE, TILE + 1, 2 * TILE + 12_345, 4 * TILE])
@pytest.mark.parametrize("group_tile_words", [64, 32])
@pytest.mark.parametrize("path", [ab.PATH_UNION, ab.PATH_HYBRID, ab.PATH_TILE])
@pytest.mark.parametrize("pad", [0, 1])
def test_bins_against_oracle(dev, n_ads, group_tile_words, path, pad):
    import torch
    off, ads = build(n_ads)
    n_terms = off.size - 1
    ix = Index.from_csr(off, ads, n_terms, n_ads)
    ix.set_tuning(group_tile_words=group_tile_words, heavy_min_len=n_ads // 300)
    qs = queries(n_terms, 40, np.random.default_rng(n_ads))
    n_words = (n_ads + 31) // 32
    stride = (n_words + 3) // 4 * 4
    terms = np.concatenate(qs)
    qoff = np.concatenate([[0], np.cumsum([q.size for q in qs])]).astype(np.uint64)
    d_t = torch.from_numpy(terms.view(np.int32)).cuda()
    d_o = torch.from_numpy(qoff.view(np.int64)).cuda()
    whole = torch.full((len(qs) * stride + 4,), -1, dtype=torch.int32, device="cuda")  # stale bits are overwritten
    bm = whole[pad:pad + len(qs) * stride]  # pad 1: rows not 16-byte aligned
    ws = ix.workspace(len(qs), terms.size)
    ix.profile(True)
    for _ in range(2):
        ix.batch_run(ws, d_t, d_o, len(qs), bm, stride, path=path)
    ws.check()
    assert ix.profile_read()["bin_union"][0] == 2
    ix.profile(False)
    got = bm.cpu().numpy().view(np.uint32).reshape(len(qs), stride)
    for i, q in enumerate(qs):
        e = O.ids_to_bitmap(O.kway_union(off, ads, q[q < n_terms]), n_words)
        assert np.array_equal(got[i, :n_words], e), i
    ix.set_tuning(group_min_queries=0)
    bm2 = torch.empty((len(qs), stride), dtype=torch.int32, device="cuda")
    ix.batch_run(ws, d_t, d_o, len(qs), bm2, stride, path=path)
    torch.cuda.synchronize()
    assert np.array_equal(bm2.cpu().numpy().view(np.uint32)[:, :n_words], got[:, :n_words])
