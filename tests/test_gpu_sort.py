"""The radix sort behind COO loads and updates, at the edges of its forms:
one-block sorts by items per thread (1, 2, 4, 8 per 1024), tiles of 4096 keys,
and keys that fit in 64 bits together with their index (packed) or do not, in
both tiers.  Duplicate keys must keep their input order (sums in batch order,
bit-exact against the oracle)."""
import numpy as np
import pytest

from helpers import assert_content_equal, assert_layout_equal, make_pair

pytestmark = pytest.mark.gpu

M31 = (1 << 31) - 1


SIZES = [
    # one block, packed: key bits + 13 <= 64
    (1, 1, 2), (3, 2, 31), (40, 7, 1023), (40, 7, 1024), (40, 300, 1025), (500, 70_000, 2048), (500, 70_000, 2049),
    (5000, 5000, 4096), (5000, 5000, 4097), (5000, 5000, 8191),
    # tiles, packed: sizes around one and several tiles, few and many passes
    (9, 3, 8193), (9, 3, 12_288), (9, 3, 12_289), (70_000, 90_000, 4096 * 3 - 1), (70_000, 90_000, 100_000),
]
WIDE = [
    # one block, packed at exactly 64 bits
    (1 << 20, M31, 8192),
    # key bits + index bits = 65: the tiles' pair form, also for small inputs
    (1 << 20, M31, 8193), ((1 << 20) + 1, M31, 2), ((1 << 20) + 1, M31, 300_001),
]


@pytest.mark.parametrize("mode,n,m,T", [(q, *z) for z in SIZES for q in (0, 1)] + [(0, *z) for z in WIDE])
def test_stable_order(dcsr, mode, n, m, T):
    rng = np.random.default_rng(T + n)
    r = rng.integers(0, n, T).astype(np.int32)
    c = rng.integers(0, m, T).astype(np.int32)
    r[T // 2:] = r[: T - T // 2]  # every key twice, far apart in the input
    c[T // 2:] = c[: T - T // 2]
    v = rng.uniform(-1, 1, T)
    dev, orc = make_pair(dcsr, n, m, 1, mode)
    dev.from_coo(r, c, v)
    assert orc.load_coo(r, c, v) == 0
    assert_layout_equal(dev, orc, "load")
    assert_content_equal(dev, orc, "load")
    if n > 100_000:  # (the oracle's wide matrices are slow: one sort each)
        return
    assert dev.update(r, c, v) == orc.update_auto(r, c, v) == 0
    assert_layout_equal(dev, orc, "update")
    assert_content_equal(dev, orc, "update")
