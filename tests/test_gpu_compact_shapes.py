"""Compaction at the edges of its chunk sizes (8, 2 or 1 units of 32 words per
warp, by the number of chunks), of the 128-byte lines its ids leave in, and of
a short output: ids, offsets and the words around the output, bit for bit."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index

pytestmark = pytest.mark.gpu

CHUNK = 1024 * 32  # ads of a chunk of 8 units per warp
FEW = 888          # chunks from which on they have 8 units (then 2, of a quarter)


def bitmap(n_bits, seed):
    """Stretches of words that are empty, full, nearly full, sparse and half full, of ragged lengths."""
    rng = np.random.default_rng(seed)
    n = (n_bits + 31) // 32
    w = np.zeros(n, np.uint32)
    i = 0
    while i < n:
        k = min(n - i, int(rng.integers(1, 700)))
        r = rng.integers(0, 1 << 32, (4, k), dtype=np.uint64).astype(np.uint32)
        w[i:i + k] = [np.zeros(k, np.uint32), np.full(k, 0xFFFFFFFF, np.uint32), r[0] | r[1] | r[2] | r[3],
                      r[0] & r[1] & r[2] & r[3], r[0]][int(rng.integers(0, 5))]
        i += k
    return w  # bits past n_bits are ignored


def ids_of(w, n_bits):
    return np.flatnonzero(np.unpackbits(w.view(np.uint8), bitorder="little")[:n_bits]).astype(np.uint32)


@pytest.fixture(scope="module")
def ix(dev):
    return Index.from_csr(np.array([0, 1], np.uint64), np.array([0], np.uint32), 1, 3 * CHUNK + 77)


@pytest.mark.parametrize("n_bits", [77, CHUNK // 8, CHUNK // 8 + 1, (FEW - 1) * CHUNK // 4 + 5, FEW * CHUNK // 4,
                                    (FEW - 1) * CHUNK - 3, (FEW - 1) * CHUNK + 1])
@pytest.mark.parametrize("shift", [0, 1, 3, 31])
@pytest.mark.parametrize("room", ["all", "short"])
def test_one_bitmap(ix, n_bits, shift, room):
    import torch
    w = bitmap(n_bits, n_bits + shift)
    want = ids_of(w, n_bits)
    cap = want.size if room == "all" else want.size // 2 + 1
    buf = torch.full((shift + want.size + 64,), -7, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    bm = torch.from_numpy(w.view(np.int32)).cuda()
    for _ in range(2):
        ab.CollectIdsFromBitmap(ix, bm, n_bits, buf[shift:shift + cap], cnt)
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    assert cnt.item() == want.size
    assert np.array_equal(got[shift:shift + min(cap, want.size)].view(np.uint32), want[:cap])
    assert np.all(got[:shift] == -7) and np.all(got[shift + min(cap, want.size):] == -7)


@pytest.mark.parametrize("n", [1, 55, 56, 221, 222, 223])  # 4 chunks of 8 units per bitmap, 13 of 2
@pytest.mark.parametrize("shift", [0, 5])
def test_batch(ix, n, shift):
    import torch
    n_words = ix.n_words
    stride = (n_words + 3) // 4 * 4 + 4
    w = np.zeros((n, stride), np.uint32)
    for i in range(n):
        w[i, :n_words] = bitmap(ix.n_ads, 1000 + i)
    want = [ids_of(w[i, :n_words], ix.n_ads) for i in range(n)]
    total = sum(a.size for a in want)
    buf = torch.full((shift + total + 64,), -7, dtype=torch.int32, device="cuda")
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ws = ix.workspace(n, 1)
    bm = torch.from_numpy(w.view(np.int32)).cuda()
    for _ in range(2):
        ab.BatchCollectIds(ix, ws, bm, stride, n, buf[shift:shift + total], off)
    ws.check()
    got, o = buf.cpu().numpy(), off.cpu().numpy()
    assert np.array_equal(o, np.concatenate([[0], np.cumsum([a.size for a in want])]))
    assert np.array_equal(got[shift:shift + total].view(np.uint32), np.concatenate(want))
    assert np.all(got[:shift] == -7) and np.all(got[shift + total:] == -7)
