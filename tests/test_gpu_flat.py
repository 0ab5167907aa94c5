"""The entry-parallel copies (CSR load, export, compaction) at the edges of
their tiles of 256 entries: entry counts around a multiple of the tile, rows
ending exactly on one, rows over many tiles, stretches of empty rows within
and past the 512 rows a tile walks before it searches instead, and rows in
several segments; layout, structure and values bit-exact against the oracle."""
import numpy as np
import pytest

import torch

from helpers import assert_content_equal, assert_layout_equal, make_pair, spmv_bound

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


def check_rows(dcsr, dev, orc, rng, what):
    """SpMV with one right-hand side (unit stride, strided, alpha and beta) and
    the row reductions against the FP64 oracle: |error| within 1e-6 (FP32) or
    1e-13 (FP64) of the sum of magnitudes."""
    tol = {0: 1e-6, 1: 1e-13}[dev.dtype_code]
    n, m = dev.n_rows, dev.n_cols
    x = torch.tensor(rng.uniform(-1, 1, (m, 3)), dtype=dev.dtype).cuda()
    y0 = torch.tensor(rng.uniform(-1, 1, (n, 2)), dtype=dev.dtype).cuda()
    x64, y64 = x.cpu().double().numpy(), y0.cpu().double().numpy()
    bound = spmv_bound(orc, x64[:, 0])
    y = dev.spmv(x[:, 0].contiguous()).cpu().double().numpy()
    assert np.all(np.abs(y - orc.spmv(x64[:, 0].copy())) <= tol * bound + 1e-300), what
    # strided x and y, accumulating (the C ABI's ldx / ldy)
    y = y0.clone()
    assert dcsr.lib().dcsr_spmv(dev.h, x.data_ptr(), 1, 3, y.data_ptr(), 2, -1.5, 0.25,
                                torch.cuda.current_stream().cuda_stream) == 0
    y = y.cpu().double().numpy()
    ref = orc.spmv(x64[:, 0].copy(), alpha=-1.5, beta=0.25, y=y64[:, 0].copy())
    assert np.all(np.abs(y[:, 0] - ref) <= tol * (1.5 * bound + 0.25 * np.abs(y64[:, 0])) + 1e-300), what
    np.testing.assert_array_equal(y[:, 1], y64[:, 1])
    rp, _, v = orc.export_csr()
    for op in (dcsr.REDUCE_SUM, dcsr.REDUCE_MAX, dcsr.REDUCE_MIN, dcsr.REDUCE_COUNT):
        got = dev.row_reduce(op).cpu().double().numpy()
        want = orc.row_reduce(op)
        if op == dcsr.REDUCE_SUM:
            mag = np.zeros(n)
            np.add.at(mag, np.repeat(np.arange(n), np.diff(rp)), np.abs(v))
            assert np.all(np.abs(got - want) <= tol * mag + 1e-300), what
        else:
            np.testing.assert_array_equal(got, want, err_msg=what)


@pytest.mark.parametrize("name", list(LENS))
@pytest.mark.parametrize("dtype", [0, 1])
def test_rows_over_tiles(dcsr, name, dtype):
    lens = np.asarray(LENS[name], np.int64)
    rng = np.random.default_rng(len(lens) + 1)
    n, m = len(lens), 100_003
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in lens if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, cols.size)
    vals = vals.astype(np.float32) if dtype == 0 else vals
    dev, orc = make_pair(dcsr, n, m, dtype, 0)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    check_rows(dcsr, dev, orc, rng, "loaded")
    for it in range(2):
        T = 700
        r = np.where(rng.random(T) < 0.5, rng.choice(np.repeat(np.arange(n), lens), T),
                     rng.integers(0, n, T)).astype(np.int32)
        c = rng.integers(0, m, T).astype(np.int32)
        v = rng.uniform(-1, 1, T)
        v = v.astype(np.float32) if dtype == 0 else v
        assert dev.update(r, c, v) == orc.update_auto(r, c, v.astype(np.float64)) == 0
        check_rows(dcsr, dev, orc, rng, f"update {it}")
    dev.compact()
    orc.compact()
    check_rows(dcsr, dev, orc, rng, "compacted")


def test_empty_matrix_rows(dcsr):
    """No entries: every row is written (0, or beta * y), the next state likewise."""
    rng = np.random.default_rng(3)
    dev, orc = make_pair(dcsr, 1000, 50, 1, 0)
    check_rows(dcsr, dev, orc, rng, "empty")
    dev.from_csr(np.zeros(1001, np.int32), np.zeros(0, np.int32), np.zeros(0))
    check_rows(dcsr, dev, orc, rng, "loaded empty")


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


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("lead", [0, 1, 255])
def test_rows_over_many_tiles(dcsr, lead, dtype):
    """Rows over about 16 tiles (where a thread stops adding their parts) and
    about 512 (where a warp does), side by side, starting anywhere in a tile."""
    rng = np.random.default_rng(lead)
    m = 300_000
    lens = [lead] + [t * 256 + d for t in (15, 16, 17, 18, 511, 512, 513, 514, 1000) for d in (0, 1, 255)] + [0, 3, 700 * 256]
    n = len(lens)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in lens if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, cols.size)
    vals = vals.astype(np.float32) if dtype == 0 else vals
    dev, orc = make_pair(dcsr, n, m, dtype, 0)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    check_rows(dcsr, dev, orc, rng, "loaded")
