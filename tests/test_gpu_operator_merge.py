"""Reference-shaped operators where they change kernels: runs of keys merged by
the dense group kernel or scattered, query bitmaps extracted to term lists in
windows, and the scan that answers a window whose terms do not fit. Bit-exact
against the oracle, on top of a bitmap that already holds bits."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N_ADS = 131_101  # ends inside a word and a tile


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=5003, n_ads=N_ADS, nnz=400_000, zipf_s=1.1, max_len=40_000, seed=31)
    off, ads = W.gen_lists(spec)
    lens = np.diff(off).astype(np.uint32)
    qoff, qt = W.gen_queries(W.QueriesSpec(300, "lognormal", 12.0, 1.5, 1, 600, seed=32), lens)
    qs = [qt[qoff[i]:qoff[i + 1]].copy() for i in range(300)]
    qs[1] = np.zeros(0, np.uint32)
    qs[2] = np.array([spec.n_terms - 1, spec.n_terms, 0xFFFFFFFF], np.uint32)  # ids at and past the domain
    return dict(spec=spec, off=off, ads=ads, qs=qs, n_words=(N_ADS + 31) // 32)


def want(env, q, seed_bits):
    q = q[q < env["spec"].n_terms]
    return O.ids_to_bitmap(O.kway_union(env["off"], env["ads"], q), env["n_words"]) | seed_bits


def start_bits(env, n, stride):
    rng = np.random.default_rng(4)
    b = np.zeros((n, stride), np.uint32)
    b[:, :env["n_words"] - 1] = rng.integers(0, 1 << 32, (n, env["n_words"] - 1), dtype=np.uint64).astype(np.uint32) & \
        rng.integers(0, 1 << 32, (n, env["n_words"] - 1), dtype=np.uint64).astype(np.uint32)
    return b


@pytest.mark.parametrize("dense_div", [0, 2048, None])
@pytest.mark.parametrize("group", [0, 1])
@pytest.mark.parametrize("order", ["runs", "split", "single"])
@pytest.mark.parametrize("repeat", [0, 1, 8])
def test_keys_by_run(env, dense_div, group, order, repeat):
    """repeat: at most 2,048 keys, scattered whole; more, in runs; the same eight times over, the group kernel's share.
    order: keys query by query; the same with every query's keys in two runs; keys shuffled (runs of a key or two)."""
    import torch
    spec = env["spec"]
    ix = Index.from_csr(env["off"], env["ads"], spec.n_terms, spec.n_ads, dense_div=dense_div)
    ix.set_tuning(group_min_queries=32 * group)
    qs = [q[q < spec.n_terms] for q in env["qs"][:40 if repeat else 12]]
    keys = np.concatenate(qs).astype(np.uint32)
    qidx = np.concatenate([np.full(q.size, i, np.uint32) for i, q in enumerate(qs)])
    if repeat > 1:  # enough postings in dense lists for the group kernel, and more runs than it takes
        keys, qidx = np.tile(keys, repeat), np.tile(qidx, repeat)
    assert (keys.size <= 2048) == (repeat == 0)
    if order == "split":
        at = np.argsort((np.arange(keys.size) % 2), kind="stable")
        keys, qidx = keys[at], qidx[at]
    elif order == "single":
        at = np.random.default_rng(5).permutation(keys.size)
        keys, qidx = keys[at], qidx[at]
    stride = env["n_words"] + 1  # rows not 8-byte aligned
    start = start_bits(env, len(qs), stride)
    w = ix.Prepare(keys)
    for _ in range(2):
        d = torch.from_numpy(start.view(np.int32).copy()).cuda()
        ab.BatchListUnion_sparse(w, d, torch.from_numpy(qidx.view(np.int32)).cuda(), stride * 4)
        torch.cuda.synchronize()
        got = d.cpu().numpy().view(np.uint32)
        for i, q in enumerate(qs):
            assert np.array_equal(got[i, :env["n_words"]], want(env, q, start[i, :env["n_words"]])), i
            assert got[i, -1] == 0


@pytest.mark.parametrize("batch", [1, 3, 31, 32, 256, 257, 300])
@pytest.mark.parametrize("device_side", [False, True])
def test_term_bitmaps_by_window(env, batch, device_side):
    import torch
    spec = env["spec"]
    ix = Index.from_csr(env["off"], env["ads"], spec.n_terms, spec.n_ads)
    length = (spec.n_terms + 31) // 32 * 4 + 4  # bits past n_terms, rows not 16-byte aligned
    host = np.zeros((batch, length), np.uint8)
    for i in range(batch):
        b = O.term_bitmap_bytes(env["qs"][i][env["qs"][i] < spec.n_terms], spec.n_terms, pad_to=1)
        host[i, :b.size] = b
        host[i, spec.n_terms // 8] |= 0xFF << (spec.n_terms % 8) & 0xFF  # ignored
        host[i, -1] = 0xFF
    stride = env["n_words"] + 1
    start = start_bits(env, batch, stride)
    w = ix.PrepareBatchDevice(batch, length, torch.from_numpy(host).cuda()) if device_side else \
        ix.PrepareBatch(batch, length, host)
    for _ in range(2):
        d = torch.from_numpy(start.view(np.int32).copy()).cuda()
        ab.BatchListUnion_dense(w, None, d, stride)
        torch.cuda.synchronize()
        got = d.cpu().numpy().view(np.uint32)
        for i in range(batch):
            assert np.array_equal(got[i, :env["n_words"]], want(env, env["qs"][i], start[i, :env["n_words"]])), i
            assert got[i, -1] == 0


@pytest.mark.parametrize("extra", [0, 1])
def test_term_bitmaps_at_the_room_for_terms(dev, extra):
    """33 queries of 2,048 terms fill their room exactly; with 2,049 each the room is short and the window is answered
    by the scan."""
    import torch
    n_terms, n_ads, batch = 2048 + extra, 4099, 33
    rng = np.random.default_rng(6)
    ads = rng.integers(0, n_ads, n_terms).astype(np.uint32)
    off = np.arange(n_terms + 1, dtype=np.uint64)
    ix = Index.from_csr(off, ads, n_terms, n_ads)
    n_words = (n_ads + 31) // 32
    length = (n_terms + 127) // 128 * 16
    host = np.full((batch, length), 0xFF, np.uint8)
    d = torch.zeros((batch, n_words), dtype=torch.int32, device="cuda")
    ab.BatchListUnion_dense(ix.PrepareBatch(batch, length, host), None, d, n_words)
    torch.cuda.synchronize()
    e = O.ids_to_bitmap(np.unique(ads), n_words)
    got = d.cpu().numpy().view(np.uint32)
    assert all(np.array_equal(got[i], e) for i in range(batch))
