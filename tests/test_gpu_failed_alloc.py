"""Device allocations that fail (dcsr_debug_fail_alloc): whichever allocation
of an operation it is, the operation reports DCSR_OOM, the matrix is as it was
before, and the same operation carried out again succeeds."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from helpers import assert_content_equal, make_pair

pytestmark = pytest.mark.gpu

N = 10_000  # more rows than one scan block: scans have a look-back area to allocate


def csr(rng, mean, sort=True):
    lens = rng.poisson(mean, N)
    lens[5] = 700
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.concatenate([rng.choice(N, L, replace=False) for L in lens if L]).astype(np.int32)
    if sort:
        cols = np.concatenate([np.sort(cols[rp[i]:rp[i + 1]]) for i in range(N)]).astype(np.int32)
    return rp, cols, rng.uniform(-1, 1, cols.size)


def coo(rng, T):
    return rng.integers(0, N, T).astype(np.int32), rng.integers(0, N, T).astype(np.int32), rng.uniform(-1, 1, T)


def operations():
    rng = np.random.default_rng(8)
    small, large, unsorted = csr(rng, 4.0), csr(rng, 60.0), csr(rng, 30.0, False)
    few, many = coo(rng, 2000), coo(rng, 150_000)
    x = torch.ones((N, 4), dtype=torch.float64).cuda()
    # first content, the operation on the device, the same on the oracle
    return {
        "csr_larger": (small, lambda d: d.from_csr(*large), lambda o: o.load_csr(*large)),
        "csr_smaller": (large, lambda d: d.from_csr(*small), lambda o: o.load_csr(*small)),
        "csr_unsorted": (small, lambda d: d.from_csr(*unsorted), lambda o: o.load_csr(*unsorted)),
        "coo": (small, lambda d: d.from_coo(*many), lambda o: o.load_coo(*many)),
        "coo_smaller": (large, lambda d: d.from_coo(*few), lambda o: o.load_coo(*few)),
        "update": (small, lambda d: d.update(*few), lambda o: o.update_auto(*few)),
        "compact": (large, lambda d: d.compact(), lambda o: o.compact()),
        "export": (large, lambda d: (d.update(*few), d.to_csr()), lambda o: o.update_auto(*few)),
        "spmv": (large, lambda d: (d.spmv(x[:, 0].contiguous()), d.spmv(x)), lambda o: None),
        "product": (small, None, None),
    }


@pytest.mark.parametrize("name", ["csr_larger", "csr_smaller", "csr_unsorted", "coo", "coo_smaller", "update", "compact",
                                  "export", "spmv", "product"])
def test_every_allocation_once(dcsr, name):
    first, run, ref = operations()[name]
    failed = 0
    for nth in range(1, 60):
        dev, orc = make_pair(dcsr, N, N, 1, 0)
        dev.from_csr(*first)
        assert orc.load_csr(*first) == 0
        if name == "product":  # into a matrix that holds something else
            rng = np.random.default_rng(9)
            a, a_o = make_pair(dcsr, N, N, 1, 0)
            rp, cols, vals = csr(rng, 12.0)
            a.from_csr(rp, cols, vals)
            assert a_o.load_csr(rp, cols, vals) == 0
            run = lambda d: a.spgemm(a, d)
        dcsr.debug_fail_alloc(nth)
        try:
            run(dev)
            ok = True
        except dcsr.DcsrError as e:
            assert e.status == dcsr.OOM
            ok = False
        finally:
            dcsr.debug_fail_alloc(0)
        if ok:
            break
        failed += 1
        if name != "export":
            assert_content_equal(dev, orc, f"{name}: allocation {nth} failed")
            run(dev)
    if name == "product":
        rp, c, v = dev.to_csr()
        rp_o, c_o, v_o = a_o.export_csr()
        m = sp.csr_matrix((v_o, c_o, rp_o), shape=(N, N))
        got = sp.csr_matrix((v.cpu().numpy(), c.cpu().numpy(), rp.cpu().numpy()), shape=(N, N))
        assert abs(got - m @ m).max() < 1e-10
    else:
        ref(orc)
        assert_content_equal(dev, orc, name)
    assert ok and (failed > 0 or name == "compact")
