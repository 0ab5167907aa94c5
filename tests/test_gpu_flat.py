"""The entry-parallel copies (CSR load, export, compaction) at the edges of
their tiles of 256 entries: entry counts around a multiple of the tile, rows
ending exactly on one, rows over many tiles, stretches of empty rows within
and past the 512 rows a tile walks before it searches instead, and rows in
several segments; layout, structure and values bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_content_equal, assert_layout_equal, make_pair

pytestmark = pytest.mark.gpu

LENS = {
    "one_entry": [0] * 5 + [1] + [0] * 7,
    "tile_less_one": [255],
    "tile": [256],
    "tile_and_one": [257],
    "rows_end_on_tiles": [256, 128, 128, 0, 255, 1, 512, 3],
    "empty_walked": [3] + [0] * 500 + [300] + [0] * 200 + [5],
    "empty_searched": [100] + [0] * 513 + [100] + [0] * 5000 + [60, 1] + [0] * 3000,
    "sparse": [1 if i % 40 == 0 else 0 for i in range(30_000)],
    "hub_rows": [70_000, 2, 0, 9_000, 4097, 1] + [3] * 100,
    "mixed": list(np.random.default_rng(7).zipf(1.6, 3000).clip(0, 5000) - 1),
}


@pytest.mark.parametrize("name", list(LENS))
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_load_export_compact(dcsr, name, dtype, mode):
    lens = np.asarray(LENS[name], np.int64)
    rng = np.random.default_rng(len(lens))
    n, m = len(lens), 100_003
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in lens if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, cols.size)
    vals = vals.astype(np.float32) if dtype == 0 else vals
    dev, orc = make_pair(dcsr, n, m, dtype, mode)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    assert_layout_equal(dev, orc, "load")
    assert_content_equal(dev, orc, "load")
    rows = np.repeat(np.arange(n), lens)
    for it in range(3):  # chained segments: triples in the longest rows and at random
        T = 700
        r = np.where(rng.random(T) < 0.5, rng.choice(rows, T), rng.integers(0, n, T)).astype(np.int32)
        c = rng.integers(0, m, T).astype(np.int32)
        v = rng.uniform(-1, 1, T)
        v = v.astype(np.float32) if dtype == 0 else v
        assert dev.update(r, c, v) == orc.update_auto(r, c, v.astype(np.float64)) == 0
        assert_layout_equal(dev, orc, f"update {it}")
        assert_content_equal(dev, orc, f"update {it}")
    rc, cc, vc = (t.cpu().numpy() for t in dev.to_coo())
    rp_o, c_o, v_o = orc.export_csr()
    np.testing.assert_array_equal(rc, np.repeat(np.arange(n), np.diff(rp_o)))
    np.testing.assert_array_equal(cc, c_o)
    np.testing.assert_array_equal(vc.astype(np.float64), v_o)
    dev.compact()
    orc.compact()
    assert_layout_equal(dev, orc, "compaction")
    assert_content_equal(dev, orc, "compaction")


@pytest.mark.parametrize("nnz", [1, 255, 256, 257, 4096, 70_001])
@pytest.mark.parametrize("at", ["first", "middle", "last", "window"])
def test_csr_check_finds_one_fault(dcsr, nnz, at):
    """The entry-parallel input check: one descent inside a row (sorted and
    summed instead), one column out of range and one negative column (refused,
    the content kept), wherever they are."""
    rng = np.random.default_rng(nnz)
    n, m = 37, 200_000
    cuts = np.sort(rng.integers(0, nnz + 1, n - 1))
    rp = np.concatenate([[0], cuts, [nnz]]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in np.diff(rp) if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, nnz)
    dev, orc = make_pair(dcsr, n, m, 1, 0)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals) == 0
    p = {"first": 0, "middle": nnz // 2, "last": nnz - 1, "window": min(31, nnz - 1)}[at]
    for bad in (-1, m):
        c = cols.copy()
        c[p] = bad
        with pytest.raises(dcsr.DcsrError) as e:
            dev.from_csr(rp, c, vals)
        assert e.value.status == dcsr.BAD_INDEX
        assert_content_equal(dev, orc, "kept")
    inside = np.flatnonzero(np.diff(cols) > 0)  # pairs within a row: swap one
    starts = set(rp.tolist())
    inside = [j for j in inside if j + 1 not in starts]
    if inside:
        j = min(inside, key=lambda q: abs(q - p))
        c = cols.copy()
        c[j], c[j + 1] = c[j + 1], c[j]
        dev.from_csr(rp, c, vals)
        assert orc.load_csr(rp, c, vals) == 0
        assert_layout_equal(dev, orc, "swapped")
        assert_content_equal(dev, orc, "swapped")
    short = rp.copy()
    short[-1] -= 1
    with pytest.raises(dcsr.DcsrError) as e:
        dev.from_csr(short, cols, vals)
    assert e.value.status == dcsr.BAD_ARG
