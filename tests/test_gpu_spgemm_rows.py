"""SpGEMM at the edges of its row classes: rows of exactly 1 to 4097 products,
with and without empty B rows among them, columns that just fit and just do not
fit the 32-bit sort keys, B rows in several segments: layout and values bit for
bit those of the oracle."""
import numpy as np
import pytest

from helpers import assert_content_equal, assert_layout_equal, make_pair, oracle_opts

pytestmark = pytest.mark.gpu

PRODUCTS = [0, 1, 31, 32, 33, 64, 65, 128, 129, 255, 256, 257, 300, 511, 512, 513, 700, 1023, 1024, 1025, 2048, 4096,
            4097]


@pytest.mark.parametrize("m", [700, 1 << 22, (1 << 22) + 1, (1 << 24) + 1])
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("empties", [False, True])
def test_product_counts(dcsr, m, dtype, empties):
    rng = np.random.default_rng(m + dtype)
    k = 6000  # B rows: the first 4200 of one entry, then of 0 (or 2) to 60 entries
    lens_b = np.concatenate([np.ones(4200, int), rng.choice([0, 3, 17, 60] if empties else [2, 3, 17, 60], k - 4200)])
    pool = np.unique(np.concatenate([rng.choice(m, 600, replace=False), [0, m - 1]]))  # columns that meet often
    b_rp = np.concatenate([[0], np.cumsum(lens_b)]).astype(np.int32)
    b_c = np.concatenate([np.sort(rng.choice(pool, L, replace=False)) for L in lens_b]).astype(np.int32)
    rows = []
    for want in PRODUCTS * 2:
        picks, have = [], 0
        for q in rng.permutation(np.arange(4200, k)):  # a third of the products from single entries
            if len(picks) < want // 20 and have + lens_b[q] <= want - want // 3:
                picks.append(q)
                have += lens_b[q]
        picks += list(rng.choice(4200, want - have, replace=False))
        rows.append(np.sort(np.array(picks, int)))
        assert sum(lens_b[q] for q in picks) == want
    n = len(rows)
    a_rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    a_c = np.concatenate(rows).astype(np.int32)
    f = np.float32 if dtype == 0 else np.float64
    a_v, b_v = rng.standard_normal(a_c.size).astype(f), rng.standard_normal(b_c.size).astype(f)
    dA, oA = make_pair(dcsr, n, k, dtype, 0)
    dB, oB = make_pair(dcsr, k, m, dtype, 0)
    dA.from_csr(a_rp, a_c, a_v)
    oA.load_csr(a_rp, a_c, a_v.astype(np.float64))
    dB.from_csr(b_rp, b_c, b_v)
    oB.load_csr(b_rp, b_c, b_v.astype(np.float64))
    for it in range(2):
        if it:  # B rows in several segments; the counts move off the edges
            r = rng.integers(0, k, 20_000).astype(np.int32)
            c, v = rng.choice(pool, r.size).astype(np.int32), rng.standard_normal(r.size).astype(f)
            assert dB.update(r, c, v) == oB.update_auto(r, c, v.astype(np.float64)) == 0
        dC = dA.spgemm(dB)
        oC = oA.spgemm(oB, oracle_opts(dC.opts))
        assert_layout_equal(dC, oC, f"C {it}")
        assert_content_equal(dC, oC, f"C {it}")
