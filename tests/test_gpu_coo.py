"""COO loads around the edges of warps, tiles and blocks: distinct triples, runs
of duplicates longer than a warp and a tile (summed in input order), both update
modes: layout and values bit for bit those of the oracle."""
import numpy as np
import pytest

from helpers import assert_content_equal, assert_layout_equal, make_pair

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4097, 8191, 8192, 8193, 30_000]


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("keys", ["distinct", "some", "few", "one"])
def test_load(dcsr, dtype, mode, keys):
    rng = np.random.default_rng(dtype + 2 * mode)
    n, m = 777, 1001
    for T in SIZES:
        if keys == "distinct":
            at = rng.choice(n * m, T, replace=False)
        elif keys == "some":
            at = rng.integers(0, n * m, max(1, T // 2))[rng.integers(0, max(1, T // 2), T)]
        elif keys == "few":
            at = rng.integers(0, n * m, 7)[rng.integers(0, 7, T)]
        else:
            at = np.full(T, n * m - 1)
        r, c = (at // m).astype(np.int32), (at % m).astype(np.int32)
        v = rng.standard_normal(T).astype(np.float32 if dtype == 0 else np.float64)
        dev, orc = make_pair(dcsr, n, m, dtype, mode)
        dev.from_coo(r, c, v)
        assert orc.load_coo(r, c, v) == 0
        assert_layout_equal(dev, orc, f"{T}")
        assert_content_equal(dev, orc, f"{T}")


@pytest.mark.parametrize("n", [8191, 8192, 8193, 8705, 262_143, 262_144, 262_145, 264_193])
def test_row_scans(dcsr, n):
    """Row counts where the scans over rows change form (one block, two and eight
    rows a thread): load, compaction after an update, export."""
    rng = np.random.default_rng(n)
    m, T = 500, 40_000
    at = rng.choice(n * m, T, replace=False)
    at[:3] = [0, n * m - 1, (n - 1) * m]
    at = np.unique(at)
    r, c = (at // m).astype(np.int32), (at % m).astype(np.int32)
    v = rng.standard_normal(at.size).astype(np.float32)
    dev, orc = make_pair(dcsr, n, m, 0, 0)
    dev.from_coo(r, c, v)
    assert orc.load_coo(r, c, v) == 0
    assert_layout_equal(dev, orc, "load")
    u = rng.integers(0, n, 5000).astype(np.int32), rng.integers(0, m, 5000).astype(np.int32)
    w = rng.standard_normal(5000).astype(np.float32)
    assert dev.update(*u, w) == orc.update_auto(*u, w.astype(np.float64)) == 0
    dev.compact()
    orc.compact()
    assert_layout_equal(dev, orc, "compacted")
    assert_content_equal(dev, orc, "compacted")
