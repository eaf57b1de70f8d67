"""A graph that captured a worker's calls outlives the worker: its replays
answer as before and touch nobody else's scratch, and the scratch comes back
when the graph is gone. Bit-exact against the oracle."""
import gc

import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index, workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N_ADS = 70_001
NW = (N_ADS + 31) // 32


@pytest.fixture(scope="module")
def env(dev):
    spec = W.ListsSpec(n_terms=5003, n_ads=N_ADS, nnz=200_000, zipf_s=1.1, max_len=20_000, seed=71)
    off, ads = W.gen_lists(spec)
    qoff, qt = W.gen_queries(W.QueriesSpec(256, "lognormal", 12.0, 1.5, 1, 600, seed=72), np.diff(off).astype(np.uint32))
    qs = [qt[qoff[i]:qoff[i + 1]].copy() for i in range(256)]
    host = np.zeros((256, (spec.n_terms + 127) // 128 * 16), np.uint8)
    for i, q in enumerate(qs):
        b = O.term_bitmap_bytes(q, spec.n_terms, pad_to=1)
        host[i, :b.size] = b
    return dict(spec=spec, off=off, ads=ads, qs=qs, host=host,
                want=np.stack([O.ids_to_bitmap(O.kway_union(off, ads, q), NW) for q in qs]))


def index(env):
    return Index.from_csr(env["off"], env["ads"], env["spec"].n_terms, N_ADS)


def result(n):
    import torch
    return torch.zeros((n, NW), dtype=torch.int32, device="cuda")


def call(env, ix, kind, n, out, stream):
    """Prepares a worker and returns it with a function that runs it."""
    import torch
    if kind == "device":
        up = torch.from_numpy(env["host"][:n]).cuda()
        torch.cuda.synchronize()
        w = ix.PrepareBatchDevice(n, env["host"].shape[1], up)
        return w, up, lambda: ab.BatchListUnion_dense(w, stream, out, NW)
    if kind == "host":
        w = ix.PrepareBatch(n, env["host"].shape[1], env["host"][:n])
        return w, None, lambda: ab.BatchListUnion_dense(w, stream, out, NW)
    keys = np.concatenate(env["qs"][:n])
    qidx = torch.from_numpy(np.repeat(np.arange(n, dtype=np.int32), [q.size for q in env["qs"][:n]])).cuda()
    w = ix.Prepare(keys)
    return w, qidx, lambda: ab.BatchListUnion_sparse(w, out, qidx, NW * 4, stream=stream)


def check(out, want):
    import torch
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("n", [1, 40, 256])
@pytest.mark.parametrize("kind", ["device", "host", "keys"])
def test_replay_after_the_worker_is_freed(env, kind, n):
    import torch
    ix = index(env)
    s = torch.cuda.Stream()
    out, other = result(n), result(n)
    w, keep, run = call(env, ix, kind, n, out, s)
    run()  # kernels loaded, lazily set attributes set
    check(out, env["want"][:n])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        run()
    w.free()
    # the next workers and a workspace of about the same sizes, alive over the replays
    later = [call(env, ix, k, n, other, s) for k in ("keys", "device", "host", "keys")]
    ws = ix.workspace(n, max(1, int(sum(q.size for q in env["qs"][:n]))))
    for _, _, again in later:
        for _ in range(2):
            out.zero_()
            torch.cuda.synchronize()
            g.replay()
            check(out, env["want"][:n])
        other.zero_()
        torch.cuda.synchronize()
        again()
        check(other, env["want"][:n])
    ws.free()
    del g, later


def test_scratch_comes_back_with_the_graph(env):
    import torch
    ix = index(env)
    s = torch.cuda.Stream()
    out = result(256)

    def one():
        w, keep, run = call(env, ix, "device", 256, out, s)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            run()
        w.free()
        g.replay()
        torch.cuda.synchronize()
        g.reset()

    for _ in range(3):
        one()
    gc.collect()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(30):  # 11 MB of scratch each
        one()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 100 << 20
    check(out, env["want"])


def test_index_freed_before_its_graph_and_worker(env):
    import torch
    for worker_first in (True, False):
        ix = index(env)
        s = torch.cuda.Stream()
        out = result(8)
        w, keep, run = call(env, ix, "device", 8, out, s)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            run()
        g.replay()
        check(out, env["want"][:8])
        if worker_first:
            w.free()
        ix.free()
        if not worker_first:
            w.free()
        g.reset()
        torch.cuda.synchronize()
