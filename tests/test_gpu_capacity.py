"""Layouts beyond the pool's index range: options whose row capacities add up
past 2^31, 2^32 and 2^48 entries are refused by every operation that lays rows
out, and leave the matrix as it was."""
import numpy as np
import pytest

import torch

from helpers import assert_content_equal, make_pair

pytestmark = pytest.mark.gpu

# rows x capacity of an empty row: 2^31, 2^32, 2^48 and a little more than each
CASES = [(1 << 18, 1 << 13), (1 << 18, 1 << 14), (1 << 18, 1 << 30), ((1 << 18) + 77, 1 << 30), (1 << 19, 1 << 29)]


@pytest.mark.parametrize("n,align", CASES)
def test_load_refused(dcsr, n, align):
    rng = np.random.default_rng(3)
    dev, orc = make_pair(dcsr, n, 1000, 1, 0, align=align)
    rp = np.zeros(n + 1, np.int32)
    rp[1 + n // 2:] = 2
    with pytest.raises(dcsr.DcsrError) as e:
        dev.from_csr(rp, np.array([3, 5], np.int32), np.array([1.0, 2.0]))
    assert e.value.status == dcsr.OOM
    T = 20_000
    with pytest.raises(dcsr.DcsrError) as e:
        dev.from_coo(rng.integers(0, n, T).astype(np.int32), rng.integers(0, 1000, T).astype(np.int32), rng.uniform(-1, 1, T))
    assert e.value.status == dcsr.OOM
    assert_content_equal(dev, orc, "refused loads")


@pytest.mark.parametrize("n,align", CASES)
def test_update_refused(dcsr, n, align):
    """One triple per row: the new segments' capacities of the whole update."""
    dev, orc = make_pair(dcsr, n, 1000, 1, 0, align=align)
    s = torch.cuda.current_stream().cuda_stream
    r = torch.arange(n, dtype=torch.int32).cuda()
    c = torch.full((n,), 7, dtype=torch.int32).cuda()
    v = torch.ones(n, dtype=torch.float64).cuda()
    assert dcsr.lib().dcsr_update(dev.h, r.data_ptr(), c.data_ptr(), v.data_ptr(), n, s) == 0
    assert dev.get_status() == dcsr.POOL_EXHAUSTED
    assert_content_equal(dev, orc, "refused update")


@pytest.mark.parametrize("n,align", CASES)
def test_product_refused(dcsr, n, align):
    a, _ = make_pair(dcsr, n, n, 1, 0)
    rp = np.minimum(np.arange(n + 1), 50).astype(np.int32)
    a.from_csr(rp, np.arange(50, dtype=np.int32), np.ones(50))
    c, orc = make_pair(dcsr, n, n, 1, 0, align=align)
    with pytest.raises(dcsr.DcsrError) as e:
        a.spgemm(a, c)
    assert e.value.status == dcsr.OOM
    assert_content_equal(c, orc, "refused product")
