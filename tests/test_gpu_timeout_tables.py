"""Row tables whose scan gave up a look-back wait (see test_gpu_timeout for the
hook): the passes behind it use none of its offsets.

The tables of the tiled passes (offsets, tile rows) are marked with a negative
entry count, the k >= 2 schedule with empty lists, before the kernels that
follow on the device read them; so SpMV, reductions and export may run while
the hook is on: they write no entry, report DCSR_TIMEOUT and leave the matrix
as it was."""
import numpy as np
import pytest
import torch

from helpers import assert_content_equal, assert_layout_equal, make_pair

pytestmark = pytest.mark.gpu

N = 20_000  # more rows than one scan block


@pytest.fixture
def pair(dcsr):
    rng = np.random.default_rng(4)
    lens = rng.poisson(6.0, N)
    lens[rng.choice(N, 40, replace=False)] = 900  # medium and long rows
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(N, L, replace=False)) for L in lens if L]).astype(np.int32)
    vals = rng.uniform(-1, 1, cols.size)
    dev, orc = make_pair(dcsr, N, N, dcsr.F64, 0)
    dev.from_csr(rp, cols, vals)
    assert orc.load_csr(rp, cols, vals) == 0
    return dev, orc


def small_update(dev, orc, seed):
    """A few triples (no look-back scan of their own): every table is stale."""
    rng = np.random.default_rng(seed)
    r, c, v = rng.integers(0, N, 50).astype(np.int32), rng.integers(0, N, 50).astype(np.int32), rng.uniform(-1, 1, 50)
    assert dev.update(r, c, v) == orc.update_auto(r, c, v) == 0


def stalled(dcsr, dev, call):
    before = dcsr.spin_faults()
    dcsr.debug_lookback(2048, True)
    try:
        call()
        torch.cuda.synchronize()
    finally:
        dcsr.debug_lookback(0, False)
    assert dcsr.spin_faults() > before


def operations(dcsr, dev):
    """Each operation on the tables, with the buffers it would write entries to."""
    s = torch.cuda.current_stream().cuda_stream
    nnz = dev.nnz() + 100  # (room for the update that follows)
    rp = torch.full((N + 1,), -7, dtype=torch.int32).cuda()
    ec = torch.full((nnz,), -7, dtype=torch.int32).cuda()
    ev = torch.full((nnz,), -7.0, dtype=torch.float64).cuda()
    x = torch.ones((N, 2), dtype=torch.float64).cuda()
    y = torch.full((N, 2), -7.0, dtype=torch.float64).cuda()
    L = dcsr.lib()
    return {
        "csr": lambda: L.dcsr_to_csr(dev.h, rp.data_ptr(), ec.data_ptr(), ev.data_ptr(), s),
        "coo": lambda: L.dcsr_to_coo(dev.h, ec.data_ptr(), ec.data_ptr(), ev.data_ptr(), s),
        "spmv": lambda: L.dcsr_spmv(dev.h, x.data_ptr(), 1, 2, y.data_ptr(), 2, 1.0, 0.0, s),
        "spmv2": lambda: L.dcsr_spmv(dev.h, x.data_ptr(), 2, 2, y.data_ptr(), 2, 1.0, 0.0, s),
        "sum": lambda: L.dcsr_row_reduce(dev.h, dcsr.REDUCE_SUM, y.data_ptr(), s),
        "bins": lambda: L.dcsr_bin_rows(dev.h, s),
    }, ec, ev


@pytest.mark.parametrize("op", ["csr", "coo", "spmv", "spmv2", "sum", "bins"])
def test_bad_tables_are_not_used(dcsr, pair, op):
    dev, orc = pair
    small_update(dev, orc, 1)
    ops, ec, ev = operations(dcsr, dev)
    small_update(dev, orc, 2)
    stalled(dcsr, dev, lambda: ops[op]())
    assert dev.get_status() == dcsr.TIMEOUT
    if op in ("csr", "coo"):
        assert bool((ec == -7).all()) and bool((ev == -7.0).all())
    small_update(dev, orc, 3)
    assert_layout_equal(dev, orc, op)
    assert_content_equal(dev, orc, op)
    x = torch.ones(N, dtype=torch.float64).cuda()
    np.testing.assert_allclose(dev.spmv(x).cpu().numpy(), orc.spmv(np.ones(N)), rtol=0, atol=1e-10)


@pytest.mark.parametrize("op", ["csr", "spmv", "spmv2", "sum", "bins"])
def test_tables_are_rebuilt_after_a_timeout(dcsr, pair, op):
    """Once the timeout has been read, export, entry count, SpMV and reductions
    build their tables anew: no update is needed in between."""
    dev, orc = pair
    small_update(dev, orc, 1)
    ops, _, _ = operations(dcsr, dev)
    small_update(dev, orc, 2)
    stalled(dcsr, dev, lambda: ops[op]())
    assert dev.get_status() == dcsr.TIMEOUT
    assert dev.nnz() == orc.export_csr()[1].size
    assert_content_equal(dev, orc, op)
    rng = np.random.default_rng(9)
    for k in (1, 2):
        x = rng.uniform(-1, 1, (N, k))
        got = dev.spmv(torch.tensor(x if k > 1 else x[:, 0].copy()).cuda()).cpu().numpy().reshape(N, k)
        for j in range(k):
            np.testing.assert_allclose(got[:, j], orc.spmv(x[:, j].copy()), rtol=0, atol=1e-10)
    np.testing.assert_allclose(dev.row_reduce(dcsr.REDUCE_SUM).cpu().numpy(), orc.row_reduce(0), rtol=0, atol=1e-10)
    assert dev.get_status() == dcsr.OK
