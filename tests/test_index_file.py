"""Damaged index files are refused, field by field, before anything is built on
them: a file that loads keeps every kernel inside its arrays."""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import Index

N_TERMS, N_ADS = 60, 100_003
ABF_ERR_IO = 6
HEADER = np.dtype([("magic", "S8"), ("version", "<u4"), ("block", "<u4"), ("n_terms", "<u4"), ("n_ads", "<u4"),
                   ("n_postings", "<u8"), ("n_blocks", "<u8"), ("n_units", "<u8"), ("max_list_len", "<u4"),
                   ("pad", "<u4")])


def lists():
    """Lists of 0, 1, 2, 127 .. 129 and more ids: random, consecutive (no payload) and far apart (wide gaps)."""
    rng = np.random.default_rng(77)
    out = [np.array([], np.uint32), np.array([N_ADS - 1], np.uint32), np.array([0, N_ADS - 1], np.uint32),
           np.arange(300, 300 + 128, dtype=np.uint32), np.arange(0, N_ADS, 781, dtype=np.uint32)]
    for n in (127, 128, 129, 255, 256, 257, 5000):
        out.append(np.sort(rng.choice(N_ADS, n, replace=False)).astype(np.uint32))
    while len(out) < N_TERMS:
        out.append(np.sort(rng.choice(N_ADS, int(rng.integers(0, 400)), replace=False)).astype(np.uint32))
    off = np.concatenate([[0], np.cumsum([x.size for x in out])]).astype(np.uint64)
    return off, np.concatenate(out).astype(np.uint32)


@pytest.fixture(scope="module")
def saved(tmp_path_factory):
    off, ads = lists()
    p = tmp_path_factory.mktemp("idx") / "good.abf"
    Index.from_csr(off, ads, N_TERMS, N_ADS, host_only=True).save(p)
    return p.read_bytes(), off, ads


def fields(raw):
    """The file's arrays, writable, over one copy of its bytes."""
    buf = bytearray(raw)
    h = np.frombuffer(buf, HEADER, 1)
    at, f = HEADER.itemsize, {"h": h}
    nt, nb, nu = int(h["n_terms"][0]), int(h["n_blocks"][0]), int(h["n_units"][0])
    for name, n in (("term_blk", nt + 1), ("term_len", nt), ("blk_first", nb), ("blk_last", nb), ("blk_term", nb),
                    ("desc", 2 * nb), ("payload", 4 * nu)):
        f[name] = np.frombuffer(buf, "<u4", n, at)
        at += 4 * n
    assert at == len(buf)
    return buf, f


def long_term(f):
    return int(np.argmax(f["term_len"]))


def packed_block(f):
    """A block with payload, not its list's last."""
    b = int(f["term_blk"][long_term(f)])
    assert f["desc"][2 * b + 1] & 63
    return b


def term_len_more(f): f["term_len"][long_term(f)] += 128
def term_len_past_the_ads(f): f["term_len"][3] = 500_000
def term_len_less(f): f["term_len"][long_term(f)] = 300
def term_len_of_an_empty_list(f): f["term_len"][0] = 1
def block_of_another_term(f): f["blk_term"][packed_block(f)] = 0
def table_gives_a_block_away(f): f["term_blk"][long_term(f)] += 1
def inner_block_short(f): f["desc"][2 * packed_block(f) + 1] -= 1 << 8
def first_id_moved(f): f["blk_first"][packed_block(f)] += 1
def last_id_moved(f): f["blk_last"][packed_block(f)] += 1
def bounds_swapped(f):
    b = packed_block(f)
    f["blk_first"][b], f["blk_last"][b] = f["blk_last"][b], f["blk_first"][b]
def blocks_out_of_order(f):
    b = packed_block(f)
    for a in (f["blk_first"], f["blk_last"]):
        a[b], a[b + 1] = a[b + 1], a[b]
    d = f["desc"].reshape(-1, 2)
    d[[b, b + 1]] = d[[b + 1, b]]
def payload_overwritten(f):
    d = int(f["desc"][2 * packed_block(f)])
    f["payload"][4 * d] ^= 0xffffffff
def payload_of_the_last_unit(f): f["desc"][2 * (f["desc"].size // 2 - 1)] += 1
def no_ads(f): f["h"]["n_ads"] = 0
def too_many_ads(f): f["h"]["n_ads"] = (1 << 31) + 1


DAMAGE = [term_len_more, term_len_past_the_ads, term_len_less, term_len_of_an_empty_list, block_of_another_term,
          table_gives_a_block_away, inner_block_short, first_id_moved, last_id_moved, bounds_swapped,
          blocks_out_of_order, payload_overwritten, payload_of_the_last_unit, no_ads, too_many_ads]


def test_undamaged_file_loads(saved, tmp_path):
    raw, off, ads = saved
    buf, _ = fields(raw)
    (tmp_path / "same.abf").write_bytes(bytes(buf))
    ix = Index.load(tmp_path / "same.abf", host_only=True)
    for t in range(N_TERMS):
        assert np.array_equal(ix.decode_list(t), ads[off[t]:off[t + 1]])


@pytest.mark.parametrize("damage", DAMAGE, ids=lambda f: f.__name__)
def test_damaged_file_is_refused(saved, tmp_path, damage):
    buf, f = fields(saved[0])
    damage(f)
    assert bytes(buf) != saved[0]
    (tmp_path / "bad.abf").write_bytes(bytes(buf))
    with pytest.raises(ab.AbfError) as e:
        Index.load(tmp_path / "bad.abf", host_only=True)
    assert e.value.status == ABF_ERR_IO
