"""SpMV with 2 to 8 right-hand sides over every row class and its edges, with
packed, strided and misaligned x (the 16-byte loads and the value-by-value
path), alpha and beta, rows in one and several segments: within 1e-6 (FP32) or
1e-13 (FP64) of the sum of magnitudes of the FP64 oracle."""
import numpy as np
import pytest
import torch

from helpers import make_pair, spmv_bound

pytestmark = pytest.mark.gpu

LENS = [0, 1, 5, 31, 32, 33, 63, 64, 65, 100, 255, 300, 511, 512, 513, 2047, 2048, 2049, 9000] + [3] * 50 + [40] * 70


@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("layout", ["packed", "strided", "misaligned"])
def test_right_hand_sides(dcsr, k, dtype, layout):
    rng = np.random.default_rng(k)
    n, m = len(LENS), 20_000
    rp = np.concatenate([[0], np.cumsum(LENS)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in LENS if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, cols.size)
    vals = vals.astype(np.float32) if dtype == 0 else vals
    dev, orc = make_pair(dcsr, n, m, dtype, 0, reloc_min=1 << 20)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals.astype(np.float64)) == 0
    tol = {0: 1e-6, 1: 1e-13}[dtype]
    ldx, ldy, off = {"packed": (k, k, 0), "strided": (k + 1, k + 2, 0), "misaligned": (k, k, 1)}[layout]
    for it in range(2):
        if it:  # rows in several segments
            r = np.repeat(np.arange(n), 60).astype(np.int32)
            c = rng.integers(0, m, r.size).astype(np.int32)
            v = rng.uniform(-1, 1, r.size)
            v = v.astype(np.float32) if dtype == 0 else v
            assert dev.update(r, c, v) == orc.update_auto(r, c, v.astype(np.float64)) == 0
        xb = torch.tensor(rng.uniform(-1, 1, m * ldx + off), dtype=dev.dtype).cuda()
        yb = torch.tensor(rng.uniform(-1, 1, n * ldy), dtype=dev.dtype).cuda()
        x = xb[off:].view(m, ldx)[:, :k].cpu().double().numpy()
        y0 = yb.view(n, ldy).cpu().double().numpy()
        bound = spmv_bound(orc, x, k)
        for alpha, beta in ((1.0, 0.0), (-0.5, 0.25)):
            y = yb.clone()
            assert dcsr.lib().dcsr_spmv(dev.h, xb[off:].data_ptr(), k, ldx, y.data_ptr(), ldy, alpha, beta,
                                        torch.cuda.current_stream().cuda_stream) == 0
            got = y.view(n, ldy).cpu().double().numpy()
            ref = orc.spmv(x.reshape(-1).copy(), k=k, alpha=alpha, beta=beta, y=y0[:, :k].reshape(-1).copy())
            err = np.abs(got[:, :k] - ref.reshape(n, k))
            lim = tol * (abs(alpha) * bound.reshape(n, k) + abs(beta) * np.abs(y0[:, :k])) + 1e-300
            assert np.all(err <= lim), f"it {it} alpha {alpha}: {np.max(err / lim):.3g}"
            np.testing.assert_array_equal(got[:, k:], y0[:, k:])


@pytest.mark.parametrize("dtype", [0, 1])
def test_classes_across_a_batch(dcsr, dtype):
    """Long, medium and short rows first and last in their matrices, matrices
    whose rows start anywhere in a block of the schedule's scan, thousands of
    long rows: a batch's results are the single calls', bit for bit."""
    rng = np.random.default_rng(5)
    sizes = [1, 2, 255, 256, 257, 2047, 2048, 2049, 1, 5000]
    work, want = [], []
    for q, n in enumerate(sizes):
        m, k = 3000, 2 + q % 7
        lens = rng.choice([0, 1, 4, 31, 40, 70, 600], n, p=[0.2, 0.3, 0.2, 0.1, 0.1, 0.05, 0.05])
        lens[0], lens[-1] = ([2500, 40], [64, 2049], [3, 700])[q % 3]
        rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in lens]).astype(np.int32)
        vals = rng.uniform(-1, 1, cols.size)
        vals = vals.astype(np.float32) if dtype == 0 else vals
        pair = []
        for _ in range(2):
            A, _orc = make_pair(dcsr, n, m, dtype, 0)
            A.set_row_classes(32, 256)
            A.from_csr(rp, cols, vals)
            pair.append(A)
        x = torch.tensor(rng.uniform(-1, 1, (m, k)), dtype=pair[0].dtype).cuda()
        work.append(dict(matrix=pair[0], x=x, y=torch.zeros(n, k, dtype=x.dtype, device="cuda")))
        want.append(pair[1].spmv(x))
    batch = dcsr.DcsrBatch(work)
    for _ in range(2):
        for w in work:
            w["y"].fill_(7)
        batch.run()
        torch.cuda.synchronize()
        for q, w in enumerate(work):
            assert torch.equal(w["y"], want[q].view_as(w["y"])), f"matrix {q}"
    batch.close()


@pytest.mark.parametrize("k", [2, 4, 6, 8])
@pytest.mark.parametrize("off", [0, 1, 2, 4])
@pytest.mark.parametrize("dtype", [0, 1])
def test_packed_rows_of_every_alignment(dcsr, k, off, dtype):
    """Packed x at each multiple of a value: rows read in vectors of 16 or 8
    bytes, or value by value, give the same sums in the same order."""
    rng = np.random.default_rng(k)
    n, m = len(LENS), 9100
    rp = np.concatenate([[0], np.cumsum(LENS)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(m, L, replace=False)) for L in LENS if L]).astype(np.int32)
    dev, _ = make_pair(dcsr, n, m, dtype, 0)
    dev.from_csr(rp, cols, torch.tensor(rng.uniform(-1, 1, cols.size), dtype=dev.dtype).cuda())
    x = torch.tensor(rng.uniform(-1, 1, (m, k)), dtype=dev.dtype).cuda()
    s = torch.cuda.current_stream().cuda_stream
    wide = torch.zeros(m, k + 1, dtype=dev.dtype).cuda()
    wide[:, :k] = x
    want, y = torch.empty(n, k, dtype=dev.dtype).cuda(), torch.empty(n, k, dtype=dev.dtype).cuda()
    assert dcsr.lib().dcsr_spmv(dev.h, wide.data_ptr(), k, k + 1, want.data_ptr(), k, 1.0, 0.0, s) == 0
    xb = torch.zeros(m * k + 4, dtype=dev.dtype).cuda()
    xb[off : off + m * k] = x.reshape(-1)
    assert dcsr.lib().dcsr_spmv(dev.h, xb[off:].data_ptr(), k, k, y.data_ptr(), k, 1.0, 0.0, s) == 0
    assert torch.equal(y, want)
