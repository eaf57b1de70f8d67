"""Scratch that passes from freed workers and workspaces to new ones of other
kinds and sizes, with several threads, and a worker prepared while a stream is
captured. Bit-exact against the oracle."""
import threading

import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N_ADS = 70_001


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=5003, n_ads=N_ADS, nnz=200_000, zipf_s=1.1, max_len=20_000, seed=51)
    off, ads = W.gen_lists(spec)
    qoff, qt = W.gen_queries(W.QueriesSpec(300, "lognormal", 12.0, 1.5, 1, 600, seed=52), np.diff(off).astype(np.uint32))
    qs = [qt[qoff[i]:qoff[i + 1]].copy() for i in range(300)]
    nw = (N_ADS + 31) // 32
    return dict(spec=spec, off=off, ads=ads, qs=qs, nw=nw, want=[O.ids_to_bitmap(O.kway_union(off, ads, q), nw) for q in qs])


def bitmaps(env, q0, n):
    host = np.zeros((n, (env["spec"].n_terms + 127) // 128 * 16), np.uint8)
    for i in range(n):
        b = O.term_bitmap_bytes(env["qs"][q0 + i], env["spec"].n_terms, pad_to=1)
        host[i, :b.size] = b
    return host


def dense(env, ix, q0, n, device_side, stream):
    import torch
    host = bitmaps(env, q0, n)
    with torch.cuda.stream(stream):
        d = torch.zeros((n, env["nw"]), dtype=torch.int32, device="cuda")
        up = torch.from_numpy(host).cuda()
        stream.synchronize()
        w = ix.PrepareBatchDevice(n, host.shape[1], up) if device_side else ix.PrepareBatch(n, host.shape[1], host)
        ab.BatchListUnion_dense(w, stream, d, env["nw"])
        got = d.cpu().numpy().view(np.uint32)
    assert all(np.array_equal(got[i], env["want"][q0 + i]) for i in range(n))


def sparse(env, ix, q, stream):
    import torch
    with torch.cuda.stream(stream):
        d = torch.zeros(env["nw"], dtype=torch.int32, device="cuda")
        ab.ListUnion_sparse(ix.Prepare(env["qs"][q]), d, stream=stream)
        got = d.cpu().numpy().view(np.uint32)
    assert np.array_equal(got, env["want"][q])


@pytest.mark.parametrize("sizes", [(256, 1, 32, 300), (1, 31, 257, 8)])
def test_scratch_changes_hands(env, sizes):
    import torch
    ix = Index.from_csr(env["off"], env["ads"], env["spec"].n_terms, N_ADS)
    s = torch.cuda.Stream()
    for n in sizes:
        for device_side in (False, True):
            dense(env, ix, 0, n, device_side, s)
            sparse(env, ix, n % 300, s)
        ix.workspace(n, 4096)  # freed at once
        with torch.cuda.stream(s):
            d = torch.zeros((env["nw"] + 3) // 4 * 4, dtype=torch.int32, device="cuda")
            ix.query(env["qs"][n % 300], d, stream=s)
            assert np.array_equal(d.cpu().numpy().view(np.uint32)[:env["nw"]], env["want"][n % 300])


def test_threads_share_the_pool(env):
    import torch
    ix = [Index.from_csr(env["off"], env["ads"], env["spec"].n_terms, N_ADS)]
    bad = []

    def work(k):
        try:
            for r in range(6):
                w = [ix[0].Prepare(env["qs"][k * 8 + r]), ix[0].PrepareBatch(4 + r, (env["spec"].n_terms + 127) // 128 * 16, bitmaps(env, k, 4 + r))]
                del w
        except Exception as e:  # reported by the main thread
            bad.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad, bad
    dense(env, ix[0], 5, 40, True, torch.cuda.Stream())


def test_prepared_while_captured(env):
    import torch
    ix = Index.from_csr(env["off"], env["ads"], env["spec"].n_terms, N_ADS)
    s = torch.cuda.Stream()
    dense(env, ix, 0, 40, True, s)  # kernels loaded
    host = bitmaps(env, 40, 256)
    up = torch.from_numpy(host).cuda()
    d = torch.zeros((256, env["nw"]), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        w = ix.PrepareBatchDevice(256, host.shape[1], up)
        ab.BatchListUnion_dense(w, s, d, env["nw"])
    for _ in range(2):
        d.zero_()
        g.replay()
        torch.cuda.synchronize()
        got = d.cpu().numpy().view(np.uint32)
        assert all(np.array_equal(got[i], env["want"][40 + i]) for i in range(256))
    del g, w
