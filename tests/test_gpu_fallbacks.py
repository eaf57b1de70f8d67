"""What an index does when device memory runs short: without plain ids its mid
lists are scattered and merged, a bitmap-probe worker without scratch is answered
by the scan, and what cannot be had at all is an error after which everything
goes on. Bit-exact against the oracle.

No memory is used up: a child process runs with a shim in front of cudaMalloc
that refuses the calls a case names."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
/* calls of lo .. hi bytes are refused, `count` of them after `skip`; live bytes are kept below `room` */
static size_t lo, hi, room, live;
static int skip, count;
static struct { void* p; size_t n; } t[65536];
static void* sym(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
void shim_refuse(size_t a, size_t b, int s, int c) { lo = a; hi = b; skip = s; count = c; }
void shim_room(size_t r) { room = r ? live + r : 0; }
size_t shim_live(void) { return live; }
int shim_left(void) { return count; }
int cudaMalloc(void** p, size_t n) {
    static int (*real)(void**, size_t);
    if (!real) real = (int (*)(void**, size_t))sym("cudaMalloc");
    if (room && live + n > room) return 2;
    if (n >= lo && n <= hi && count > 0 && skip-- <= 0) { --count; return 2; }
    int e = real(p, n);
    if (!e) { size_t i = ((size_t)*p >> 8) % 65536; while (t[i].p) i = (i + 1) % 65536; t[i].p = *p; t[i].n = n; live += n; }
    return e;
}
int cudaFree(void* p) {
    static int (*real)(void*);
    if (!real) real = (int (*)(void*))sym("cudaFree");
    for (size_t i = 0; p && i < 65536; ++i) if (t[i].p == p) { live -= t[i].n; t[i].p = 0; break; }
    return real(p);
}
"""

N_ADS = 200_003
NW = (N_ADS + 31) // 32
STRIDE = (NW + 3) // 4 * 4


# ---- in the child ----------------------------------------------------------
def make():
    import torch
    import adabool_b200 as ab
    from adabool_b200 import workload as W
    from oracle import oracle as O
    torch.zeros(1, device="cuda")
    spec = W.ListsSpec(n_terms=4001, n_ads=N_ADS, nnz=900_000, zipf_s=1.1, max_len=60_000, seed=91)
    off, ads = W.gen_lists(spec)
    qoff, qt = W.gen_queries(W.QueriesSpec(300, "lognormal", 12.0, 1.5, 1, 600, seed=92), np.diff(off).astype(np.uint32))
    qs = [qt[qoff[i]:qoff[i + 1]].copy() for i in range(300)]
    want = [O.ids_to_bitmap(O.kway_union(off, ads, q), NW) for q in qs]
    return dict(ab=ab, off=off, ads=ads, spec=spec, qoff=qoff, qt=qt, qs=qs, want=want, shim=C.CDLL(None),
                build=lambda **kw: ab.Index.from_csr(off, ads, spec.n_terms, N_ADS, **kw))


def same(got, want, what):
    assert np.array_equal(got, want), what


def all_ways(e, ix, sizes=(1, 7, 40)):
    import torch
    ab = e["ab"]
    dt, do = torch.from_numpy(e["qt"].view(np.int32)).cuda(), torch.from_numpy(e["qoff"].view(np.int64)).cuda()
    for n in sizes:
        ws = ix.workspace(n, int(e["qoff"][n]))
        for path in (ab.PATH_AUTO, ab.PATH_UNION, ab.PATH_HYBRID, ab.PATH_TILE, ab.PATH_PROBE):
            bm = torch.full((n, STRIDE), -1, dtype=torch.int32, device="cuda")
            ix.batch_run(ws, dt, do, n, bm, STRIDE, path=path)
            ws.check()
            got = bm.cpu().numpy().view(np.uint32)
            for i in range(n):
                same(got[i, :NW], e["want"][i], (n, path, i))
        out = torch.zeros((n, STRIDE), dtype=torch.int32, device="cuda")
        qidx = torch.from_numpy(np.repeat(np.arange(n, dtype=np.int32), [q.size for q in e["qs"][:n]])).cuda()
        ab.BatchListUnion_sparse(ix.Prepare(np.concatenate(e["qs"][:n])), out, qidx, STRIDE * 4)
        got = out.cpu().numpy().view(np.uint32)
        for i in range(n):
            same(got[i, :NW], e["want"][i], (n, "keys", i))
    for i in range(5):
        out = torch.zeros(STRIDE, dtype=torch.int32, device="cuda")
        ab.ListUnion_sparse(ix.Prepare(e["qs"][i]), out)
        same(out.cpu().numpy().view(np.uint32)[:NW], e["want"][i], ("one", i))
    dense(e, ix, 40, True)


def dense(e, ix, n, device_side, worker=None):
    import torch
    from oracle import oracle as O
    host = np.zeros((n, (e["spec"].n_terms + 127) // 128 * 16), np.uint8)
    for i in range(n):
        b = O.term_bitmap_bytes(e["qs"][i], e["spec"].n_terms, pad_to=1)
        host[i, :b.size] = b
    up = torch.from_numpy(host).cuda()
    out = torch.zeros((n, STRIDE), dtype=torch.int32, device="cuda")
    if worker:
        worker()
    w = ix.PrepareBatchDevice(n, host.shape[1], up) if device_side else ix.PrepareBatch(n, host.shape[1], host)
    e["ab"].BatchListUnion_dense(w, None, out, STRIDE)
    got = out.cpu().numpy().view(np.uint32)
    for i in range(n):
        same(got[i, :NW], e["want"][i], ("dense", n, device_side, i))
    w.check()
    return w


def device_bytes(ix):
    return ix.stats()["device_bytes"]


def case_plain_ids_refused():
    """At the upload and when the dense bitmaps are rebuilt; the ids are the largest array without dense bitmaps."""
    e = make()
    full = e["build"](dense_div=None)
    plain = device_bytes(full)
    ids = int(np.diff(e["off"])[np.diff(e["off"]) >= 256].sum()) * 4
    e["shim"].shim_refuse(C.c_size_t(ids), C.c_size_t(ids * 3 // 2), 0, 1)
    ix = e["build"](dense_div=None)
    assert e["shim"].shim_left() == 0 and device_bytes(ix) <= plain - ids
    all_ways(e, ix)
    ix.set_tuning(heavy_min_len=256, group_min_queries=0)
    all_ways(e, ix)
    for div in (0, None):
        ix.set_dense_div(div)  # now there is room
        all_ways(e, ix, (7, 40))
    assert device_bytes(ix) >= plain
    e["shim"].shim_refuse(C.c_size_t(ids), C.c_size_t(ids * 3 // 2), 0, 1)
    ix.set_dense_div(None)
    assert e["shim"].shim_left() == 0 and device_bytes(ix) <= plain - ids
    all_ways(e, ix, (7, 40))


def case_room_for_all_but_the_plain_ids():
    """The term tables are not crowded out by the plain ids."""
    e = make()
    shim = e["shim"]
    shim.shim_live.restype = C.c_size_t
    before = shim.shim_live()
    full = e["build"]()
    used = shim.shim_live() - before
    full.free()
    assert shim.shim_live() == before
    for less in (1, 20_000, 60_000, 120_000, 300_000):  # the tables take 128 KB, the plain ids more than 1 MB
        shim.shim_room(C.c_size_t(used - less))
        ix = e["build"]()
        shim.shim_room(C.c_size_t(0))
        all_ways(e, ix, (7,))
        ix.free()


def case_worker_without_scratch():
    e = make()
    for n in (1, 33, 300):
        for device_side in (True, False):
            ix = e["build"]()  # with an empty pool of scratch
            # the lists' scratch is refused twice (once more after the pool is emptied); the bitmaps' own copy is had
            refuse = lambda: e["shim"].shim_refuse(C.c_size_t(1 << 15), C.c_size_t(1 << 40), 0, 2)
            w = dense(e, ix, n, device_side, refuse)
            assert e["shim"].shim_left() == 0
            with pytest.raises(e["ab"].AbfError):
                w.selftest_waits(1 << 12)  # it has none of that scratch
            dense(e, ix, n, device_side)
    # a sparse worker and a workspace are refused, and had the next time
    for get in (lambda: ix.Prepare(np.resize(e["qt"], 200_000)), lambda: ix.workspace(4096, 1 << 20)):
        e["shim"].shim_refuse(C.c_size_t(1 << 18), C.c_size_t(1 << 40), 0, 2)
        with pytest.raises(e["ab"].AbfError) as err:
            get()
        assert err.value.status == 4 and e["shim"].shim_left() == 0  # ABF_ERR_OOM
        get()
    all_ways(e, ix, (7, 40))


# ---- here --------------------------------------------------------------------
@pytest.fixture(scope="module")
def shim(dev, tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(d / "shim.c"), "-o", str(d / "shim.so"), "-ldl"], check=True)
    return d / "shim.so"


@pytest.mark.parametrize("case", ["plain_ids_refused", "room_for_all_but_the_plain_ids", "worker_without_scratch"])
def test_memory_runs_short(shim, case):
    root = Path(__file__).resolve().parents[1]
    env = dict(os.environ, LD_PRELOAD=str(shim), PYTHONPATH=str(root))
    r = subprocess.run([sys.executable, __file__, case], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def test_lists_past_the_plain_ids_budget(dev):
    """Plain ids stop at 256 MB: the shorter ones of 80M postings stay bare, and HYBRID merges them from blocks."""
    import torch
    import adabool_b200 as ab
    from adabool_b200 import Index, workload as W
    from oracle import oracle as O
    n_ads = 1 << 21
    spec = W.ListsSpec(n_terms=40_000, n_ads=n_ads, nnz=80_000_000, zipf_s=0.6, max_len=60_000, seed=93)
    off, ads = W.gen_lists(spec)
    lens = np.diff(off).astype(np.uint32)
    ix = Index.from_csr(off, ads, spec.n_terms, n_ads, dense_div=None)
    long = np.sort(lens[lens >= 256].astype(np.int64))[::-1]
    cut = long[np.cumsum(4 * long) > 256 << 20]
    assert cut.size > 1000 and cut[0] > 600  # bare lists that HYBRID merges below
    qoff, qt = W.gen_queries(W.QueriesSpec(40, "lognormal", 40.0, 1.0, 1, 500, seed=94), lens)
    want = [O.ids_to_bitmap(O.kway_union(off, ads, qt[qoff[i]:qoff[i + 1]]), n_ads // 32) for i in range(40)]
    dt, do = torch.from_numpy(qt.view(np.int32)).cuda(), torch.from_numpy(qoff.view(np.int64)).cuda()
    for tuning in (dict(), dict(heavy_min_len=512), dict(heavy_min_len=512, group_min_queries=0)):
        ix.set_tuning(**tuning)
        for n in (3, 40):
            ws = ix.workspace(n, qt.size)
            for path in (ab.PATH_AUTO, ab.PATH_UNION, ab.PATH_HYBRID, ab.PATH_TILE):
                bm = torch.full((n, n_ads // 32), -1, dtype=torch.int32, device="cuda")
                ix.batch_run(ws, dt, do, n, bm, n_ads // 32, path=path)
                ws.check()
                got = bm.cpu().numpy().view(np.uint32)
                assert all(np.array_equal(got[i], want[i]) for i in range(n)), (tuning, n, path)
        for i in range(4):
            out = torch.zeros(n_ads // 32, dtype=torch.int32, device="cuda")
            ab.ListUnion_sparse(ix.Prepare(qt[qoff[i]:qoff[i + 1]]), out)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want[i]), (tuning, i)


if __name__ == "__main__":
    globals()["case_" + sys.argv[1]]()
