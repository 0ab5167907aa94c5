"""In-place insertion, relocation and list edges of the update's apply step:
rows whose changed stretch is 1, 31..33, 255..257 and several times 256
positions, insertions before the first, between two and after the last entry
(many at one place), more new columns than lanes, rows in several segments,
and relocations of short, long and empty rows; bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_content_equal, assert_layout_equal, make_pair

pytestmark = pytest.mark.gpu

M = 100_000


def build(rng, lens):
    """Rows with the columns 10, 20, 30, ... so that insertions can be aimed."""
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([10 * np.arange(1, L + 1) for L in lens if L]).astype(np.int32)
    return rp, cols, rng.uniform(-1, 1, cols.size)


def aimed(rng, lens, kind):
    r, c = [], []
    for i, L in enumerate(lens):
        if kind == "front":
            k = [1 + j for j in range(1 + i % 9)]
        elif kind == "back":
            k = [10 * L + 11 + j for j in range(1 + i % 9)]
        elif kind == "one_place":
            k = [10 * (L // 2) + 1 + j for j in range(9)]
        elif kind == "spread":
            k = [10 * q + 5 for q in range(0, L + 1, max(1, L // 7))]
        elif kind == "many":
            k = [10 * q + 1 + j for q in range(0, L + 1, max(1, L // 20)) for j in range(5)]
        else:  # existing and new mixed, duplicates
            k = list(rng.integers(1, 10 * L + 30, 12)) + [10 * (1 + q % max(L, 1)) for q in range(5)] * 2
        r += [i] * len(k)
        c += k
    order = rng.permutation(len(r))
    return np.asarray(r, np.int32)[order], np.asarray(c, np.int32)[order], rng.uniform(-1, 1, len(r))


LENS = [0, 1, 2, 7, 8, 22, 23, 24, 30, 31, 32, 33, 63, 64, 95, 96, 97, 246, 247, 248, 255, 256, 257, 300, 503, 511, 512,
        513, 1000, 2047, 2048, 2049, 2600, 5000]


@pytest.mark.parametrize("kind", ["front", "back", "one_place", "spread", "many", "mixed"])
@pytest.mark.parametrize("dtype,reloc_min", [(0, 2048), (1, 2048), (0, 0), (1, 20), (1, 1 << 20)])
def test_aimed_insertions(dcsr, kind, dtype, reloc_min):
    rng = np.random.default_rng(len(kind) + reloc_min)
    lens = LENS
    rp, cols, vals = build(rng, lens)
    vals = vals.astype(np.float32) if dtype == 0 else vals
    dev, orc = make_pair(dcsr, len(lens), M, dtype, 0, reloc_min=reloc_min, min_cap=2)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    for it in range(4):  # later rounds meet rows in several segments
        r, c, v = aimed(rng, lens, kind if it % 2 == 0 else "mixed")
        c = np.minimum(c + it, M - 1).astype(np.int32)
        v = v.astype(np.float32) if dtype == 0 else v
        assert dev.update(r, c, v) == orc.update_auto(r, c, v.astype(np.float64)) == 0
        assert_layout_equal(dev, orc, f"round {it}")
        assert_content_equal(dev, orc, f"round {it}")


@pytest.mark.parametrize("T", [1, 1023, 1024, 1025, 2048, 5000])
def test_batch_sizes_around_the_scan_tiles(dcsr, T):
    rng = np.random.default_rng(T)
    n = 300
    lens = rng.integers(0, 60, n)
    rp, cols, vals = build(rng, lens)
    for mode in (0, 1):
        dev, orc = make_pair(dcsr, n, M, 1, mode)
        dev.from_csr(rp, cols, vals)
        assert orc.load_csr(rp, cols, vals) == 0
        for _ in range(2):
            r = rng.integers(0, n, T).astype(np.int32)
            c = rng.integers(0, 700, T).astype(np.int32)
            v = rng.uniform(-1, 1, T)
            assert dev.update(r, c, v) == orc.update_auto(r, c, v) == 0
            assert_layout_equal(dev, orc, f"T={T}")
            assert_content_equal(dev, orc, f"T={T}")


def grown_rows(rng, n, segs):
    """n rows of 2 to 4 entries and triples that relocate most of them: a new
    first column (reloc_min = 0), or one past each row's capacity (max_segs = 1)."""
    lens = rng.integers(2, 5, n)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([10 * np.arange(1, L + 1) for L in lens]).astype(np.int32)
    each = 1 if segs else 7
    hit = np.sort(rng.choice(n, n - n // 50, replace=False))  # some rows stay
    r = np.repeat(hit, each).astype(np.int32)
    c = (3 + np.tile(np.arange(each), hit.size) * 11 + (r % 5)).astype(np.int32)
    order = rng.permutation(r.size)
    return rp, cols, rng.uniform(-1, 1, cols.size), r[order], c[order], rng.uniform(-1, 1, r.size)


@pytest.mark.parametrize("n", [66_000, 68_000, 140_000])
@pytest.mark.parametrize("segs", [0, 1])
@pytest.mark.parametrize("dtype", [0, 1])
def test_many_relocated_rows(dcsr, n, segs, dtype):
    """More rows relocated by one update than 16 bits count (65536), and than
    twice that."""
    rng = np.random.default_rng(n + segs)
    rp, cols, vals, r, c, v = grown_rows(rng, n, segs)
    kw = dict(reloc_min=0) if segs else dict(max_segs=1)
    dev, orc = make_pair(dcsr, n, M, dtype, 0, spare_x16=64, **kw)
    ft = np.float32 if dtype == 0 else np.float64
    vals, v = vals.astype(ft), v.astype(ft)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    for it in range(2):
        assert dev.update(r, c + 60 * it, v) == orc.update_auto(r, c + 60 * it, v.astype(np.float64)) == 0
        assert_layout_equal(dev, orc, f"update {it}")
        assert_content_equal(dev, orc, f"update {it}")


def test_many_relocated_rows_batched(dcsr):
    """The same, counted over the matrices of a batch."""
    import torch
    work, orcs = [], []
    for q, n in enumerate([40_000, 66_000, 3, 50_000]):
        rng = np.random.default_rng(q)
        rp, cols, vals, r, c, v = grown_rows(rng, n, 1)
        dev, orc = make_pair(dcsr, n, M, 1, 0, spare_x16=64, reloc_min=0)
        dev.from_csr(rp, cols, vals)
        assert orc.load_csr(rp, cols, vals) == 0
        assert orc.update_auto(r, c, v) == 0
        work.append(dict(matrix=dev, rows=torch.tensor(r).cuda(), cols=torch.tensor(c).cuda(), vals=torch.tensor(v).cuda()))
        orcs.append(orc)
    batch = dcsr.DcsrBatch(work)
    batch.run()
    assert not batch.status().any()
    for w, orc in zip(work, orcs):
        assert_layout_equal(w["matrix"], orc, "batched")
        assert_content_equal(w["matrix"], orc, "batched")
    batch.close()


COUNTS = [1, 2, 3, 4, 5, 6, 7, 31, 32, 33, 35, 36, 37, 63, 64, 65, 127, 128, 129, 131, 132, 133, 134, 259, 260, 261, 1000, 20_000]


def repeated(rng, per_count, n, cols_of):
    """Triples whose (row, column) pairs come COUNTS times each."""
    r, c = [], []
    for q in range(per_count):
        for i, k in enumerate(COUNTS):
            r.append(np.full(k, (q * len(COUNTS) + 7 * i) % n))
            c.append(np.full(k, cols_of(q, i)))
    r, c = np.concatenate(r), np.concatenate(c)
    order = rng.permutation(r.size)
    return r[order].astype(np.int32), c[order].astype(np.int32), rng.uniform(-1, 1, r.size)


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("per_count", [1, 9])
def test_repeated_pairs(dcsr, dtype, per_count):
    """Pairs that come once to 20,000 times in an update, new and existing
    columns, added up in batch order, alone and in a batch."""
    import torch
    rng = np.random.default_rng(per_count)
    lens = rng.integers(0, 40, 500)
    rp, cols, vals = build(rng, lens)
    ft = np.float32 if dtype == 0 else np.float64
    dev, orc = make_pair(dcsr, 500, M, dtype, 0)
    bat, _ = make_pair(dcsr, 500, M, dtype, 0)
    for m in (dev, bat):
        m.from_csr(rp, cols, vals.astype(ft))
    assert orc.load_csr(rp, cols, vals.astype(ft).astype(np.float64)) == 0
    for it in range(3):  # the second round's pairs are all there
        r, c, v = repeated(rng, per_count, 500, lambda q, i: 10 * (1 + i % 5) if (q + i + it // 2) % 2 else 1003 + 11 * i + q)
        v = v.astype(ft)
        assert dev.update(r, c, v) == orc.update_auto(r, c, v.astype(np.float64)) == 0
        assert_layout_equal(dev, orc, f"update {it}")
        assert_content_equal(dev, orc, f"update {it}")
        batch = dcsr.DcsrBatch([dict(matrix=bat, rows=torch.tensor(r).cuda(), cols=torch.tensor(c).cuda(),
                                     vals=torch.tensor(v).cuda())])
        batch.run()
        batch.repair(batch.status())
        assert_content_equal(bat, orc, f"batched update {it}")
        batch.close()


@pytest.mark.parametrize("dtype", [0, 1])
def test_append_many_to_a_row(dcsr, dtype):
    """Append mode: rows that take one to 20,000 triples in an update, on rows of
    no, one and several segments."""
    rng = np.random.default_rng(2)
    n = 3 * len(COUNTS)
    lens = rng.integers(0, 30, n)
    rp, cols, vals = build(rng, lens)
    ft = np.float32 if dtype == 0 else np.float64
    dev, orc = make_pair(dcsr, n, M, dtype, 1)
    dev.from_csr(rp, cols, vals.astype(ft))
    assert orc.load_csr(rp, cols, vals.astype(ft).astype(np.float64)) == 0
    for it in range(3):
        r = np.concatenate([np.full(k, (3 * i + it * 5) % n) for i, k in enumerate(COUNTS)])
        r = r[rng.permutation(r.size)].astype(np.int32)
        c, v = rng.integers(0, M, r.size).astype(np.int32), rng.uniform(-1, 1, r.size).astype(ft)
        assert dev.update(r, c, v) == orc.update_auto(r, c, v.astype(np.float64)) == 0
        assert_layout_equal(dev, orc, f"append {it}")
        assert_content_equal(dev, orc, f"append {it}")


@pytest.mark.parametrize("T", [1, 20])
def test_few_triples_move_long_rows(dcsr, T):
    """One and twenty triples whose rows, of 400,000 and 1,000,000 entries,
    are relocated whole."""
    rng = np.random.default_rng(T)
    m = 3_000_000
    lens = [3, 1_000_000, 0, 400_000, 5]
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in lens if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, cols.size)
    dev, orc = make_pair(dcsr, 5, m, 1, 0)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals) == 0
    for it in range(3):
        r = (1 + 2 * (np.arange(T) % 2)).astype(np.int32)
        c, v = rng.integers(0, m, T).astype(np.int32), rng.uniform(-1, 1, T)
        assert dev.update(r, c, v) == orc.update_auto(r, c, v) == 0
        assert_layout_equal(dev, orc, f"update {it}")
        assert_content_equal(dev, orc, f"update {it}")
