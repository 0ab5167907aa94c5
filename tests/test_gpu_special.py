"""Infinities, NaNs and the ends of the exponent range in the passes over one
value per entry.

The right-hand sides and values are powers of two, infinities or NaN, so that
every sum in 64 bits is exact (or a definite infinity or NaN) in whatever order
it is taken, and results are compared for equality.  FP32 matrices of up to
32768 rows multiply in 64 bits, larger ones in 32 (the reference below does the
same).  Row maxima and minima follow the oracle: NaN when a row's first entry
is, later NaNs passed over."""
import numpy as np
import pytest
import torch

from tests.helpers import make_pair

pytestmark = pytest.mark.gpu

INF, NAN, BIG, TINY = np.inf, np.nan, 2.0**100, 2.0**-100
M = 4000  # columns: [0] inf, [1] -inf, [2] nan, [3..999] 1, [1000..1999] BIG, [2000..] TINY
X = np.ones(M)
X[:3] = INF, -INF, NAN
X[1000:2000] = BIG
X[2000:] = TINY
ONE, BIGC, TINYC = 3, 1000, 2000
SHORT = [  # rows of (column, value)
    [(0, 1.0)], [(1, 1.0)], [(2, 1.0)], [(0, 1.0), (1, 1.0)], [(0, 0.0)],
    [(ONE, INF)], [(ONE, -INF), (ONE + 1, 1.0)], [(ONE, INF), (ONE + 1, -INF)], [(ONE, NAN)],
    [(BIGC, BIG)], [(BIGC, -BIG)], [(BIGC, BIG), (BIGC + 1, -BIG)],
    [(TINYC, TINY)], [(TINYC, TINY), (TINYC + 1, TINY)], [(TINYC, TINY), (TINYC + 1, -TINY)],
    [], [(ONE, 1.0), (ONE + 1, 2.0)],
]


def rows_of(n, special):
    """The short rows, then rows over several tiles of 256 entries: all of one
    large or small product, with one special entry first, inside or last."""
    rows = [list(r) for r in SHORT] if special else [[(ONE, 1.0)]]
    for first, count, v in ((BIGC, 900, BIG), (BIGC, 900, -BIG), (TINYC, 900, TINY), (ONE, 800, 0.5)):
        rows.append([(first + j, v) for j in range(count)])
        if special:
            for at in (0, 450, count - 1):
                for sp in (INF, -INF, NAN):
                    rows.append([(first + j, sp if j == at else v) for j in range(count)])
    rows += [[] for _ in range(n - len(rows))]
    return rows


def expect(rows, dtype, n, alpha, beta, y0):
    ft = np.float32 if dtype == torch.float32 else np.float64
    pt = np.float32 if dtype == torch.float32 and n > 32768 else np.float64
    with np.errstate(all="ignore"):
        x = X.astype(ft)
        y = np.array([sum((float(pt(ft(v)) * pt(x[c])) for c, v in r), 0.0) if r else 0.0 for r in rows])
        y = y * alpha
        return (y + beta * y0.astype(np.float64) if beta else y).astype(ft)


@pytest.mark.parametrize("n", [200, 32768, 32769])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (2.0**-150, 0.0), (2.0**120, 2.0)])
def test_spmv_one_rhs(dcsr, n, dtype, alpha, beta):
    rows = rows_of(n, True)
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    cols = np.array([c for r in rows for c, _ in r], np.int32)
    vals = np.array([v for r in rows for _, v in r])
    a = dcsr.DcsrMatrix(n, M, dtype)
    a.from_csr(rp, cols, torch.tensor(vals, dtype=dtype).cuda())
    x = torch.tensor(X, dtype=dtype).cuda()
    y0 = torch.tensor(np.arange(n) % 7, dtype=dtype).cuda()
    want = expect(rows, dtype, n, alpha, beta, y0.cpu().numpy())
    y = y0.clone()
    a.spmv(x, y, alpha, beta)
    np.testing.assert_array_equal(y.cpu().numpy(), want)
    # the batched form, beside a matrix on the other side of the line
    n2 = 40_000 if n <= 32768 else 100
    rows2 = rows_of(n2, False)
    b = dcsr.DcsrMatrix(n2, M, dtype)
    b.from_csr(np.concatenate([[0], np.cumsum([len(r) for r in rows2])]).astype(np.int32),
               np.array([c for r in rows2 for c, _ in r], np.int32),
               torch.tensor([v for r in rows2 for _, v in r], dtype=dtype).cuda())
    y, y2 = y0.clone(), torch.zeros(n2, dtype=dtype).cuda()
    batch = dcsr.DcsrBatch([dict(matrix=a, x=x, y=y, alpha=alpha, beta=beta), dict(matrix=b, x=x, y=y2, alpha=alpha)])
    batch.run()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(y.cpu().numpy(), want)
    np.testing.assert_array_equal(y2.cpu().numpy(), expect(rows2, dtype, n2, alpha, 0.0, np.zeros(n2)))
    batch.close()


@pytest.mark.parametrize("dtype", [0, 1])
def test_extremes_with_nan(dcsr, dtype):
    """NaN first, inside, last and everywhere; infinities of both signs; rows
    within a lane's eight entries, over lanes, over tiles and over more than
    16 tiles, starting at every kind of place in a tile."""
    rng = np.random.default_rng(5)
    rows = []
    for L in (1, 2, 3, 7, 8, 9, 31, 33, 255, 256, 257, 700, 5000):
        for kind in ("first", "inside", "last", "all", "first_two", "minus_inf", "plus_inf", "none"):
            v = rng.uniform(-1, 1, L)
            if kind == "first":
                v[0] = NAN
            elif kind == "inside":
                v[L // 2] = NAN
            elif kind == "last":
                v[-1] = NAN
            elif kind == "all":
                v[:] = NAN
            elif kind == "first_two":
                v[: min(2, L)] = NAN
            elif kind == "minus_inf":
                v[:] = -INF
            elif kind == "plus_inf":
                v[:] = INF
            rows.append(v)
            if kind == "inside":
                rows.append(np.zeros(0))
    rows = [rows[i] for i in rng.permutation(len(rows))] + rows  # (and in a regular order)
    n, m = len(rows), 6000
    rp = np.concatenate([[0], np.cumsum([len(v) for v in rows])]).astype(np.int32)
    cols = np.concatenate([np.arange(len(v)) for v in rows]).astype(np.int32)
    vals = np.concatenate(rows)
    vals = vals.astype(np.float32) if dtype == 0 else vals
    dev, orc = make_pair(dcsr, n, m, dtype, 0)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    for op in (dcsr.REDUCE_MAX, dcsr.REDUCE_MIN):
        np.testing.assert_array_equal(dev.row_reduce(op).cpu().double().numpy(), orc.row_reduce(op))
