"""Updates, SpMVs, reductions and exports inside a caller's own stream capture
(torch.cuda.graph), and calls outside it on the same matrix: a graph's runs
change the rows unseen by the host, so whatever is read afterwards, entry
count, export, reductions, SpMV, is that of the rows as they are; and what a
call before the capture prepared is enough for the calls in it."""
import numpy as np
import pytest
import torch

from helpers import assert_content_equal, make_pair

pytestmark = pytest.mark.gpu

N = 20_000  # more rows than one scan block: tables are built with look-back


class Case:
    def __init__(self, dcsr, seed, T=600, load=True):
        self.dcsr, self.rng, self.T = dcsr, np.random.default_rng(seed), T
        self.dev, self.orc = make_pair(dcsr, N, N, dcsr.F64, 0, min_spare=1 << 20)
        if load:
            lens = self.rng.poisson(5.0, N)
            lens[self.rng.choice(N, 30, replace=False)] = 800
            rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
            cols = np.concatenate([np.sort(self.rng.choice(N, L, replace=False)) for L in lens if L]).astype(np.int32)
            vals = self.rng.uniform(-1, 1, cols.size)
            self.dev.from_csr(rp, cols, vals)
            assert self.orc.load_csr(rp, cols, vals) == 0
        self.r = torch.zeros(T, dtype=torch.int32).cuda()
        self.c, self.v = self.r.clone(), torch.zeros(T, dtype=torch.float64).cuda()
        self.x = torch.tensor(self.rng.uniform(-1, 1, (N, 4))).cuda()
        self.y = torch.zeros((N, 4), dtype=torch.float64).cuda()
        self.s = torch.cuda.Stream()

    def triples(self):
        """New triples in place, a third of them in one row; the same into the oracle."""
        r = self.rng.integers(0, N, self.T).astype(np.int32)
        r[: self.T // 3] = self.rng.integers(0, N)
        c, v = self.rng.integers(0, N, self.T).astype(np.int32), self.rng.uniform(-1, 1, self.T)
        for t, a in ((self.r, r), (self.c, c), (self.v, v)):
            t.copy_(torch.tensor(a))
        assert self.orc.update_auto(r, c, v) == 0
        torch.cuda.synchronize()

    def update(self):
        self.check(self.dcsr.lib().dcsr_update(self.dev.h, self.r.data_ptr(), self.c.data_ptr(), self.v.data_ptr(), self.T,
                                               self.s.cuda_stream))

    def spmv(self, k):
        self.check(self.dcsr.lib().dcsr_spmv(self.dev.h, self.x.data_ptr(), k, 4, self.y.data_ptr(), 4, 1.0, 0.0,
                                             self.s.cuda_stream))

    @staticmethod
    def check(status):
        assert status == 0, status

    def captured(self, *calls):
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=self.s):
            for call in calls:
                call()
        return g

    def run(self, g):
        self.triples()
        g.replay()
        torch.cuda.synchronize()

    def spmv_is_right(self, k):
        y = self.dev.spmv(self.x[:, :k].contiguous()).cpu().numpy()
        for j in range(k):
            np.testing.assert_allclose(y[:, j], self.orc.spmv(self.x[:, j].cpu().numpy().copy()), rtol=0, atol=1e-9)

    def all_right(self, what):
        assert self.dev.nnz() == self.orc.export_csr()[1].size, what
        assert_content_equal(self.dev, self.orc, what)
        for op in (self.dcsr.REDUCE_COUNT, self.dcsr.REDUCE_MAX):
            np.testing.assert_array_equal(self.dev.row_reduce(op).cpu().numpy(), self.orc.row_reduce(op), err_msg=what)
        for k in (1, 2, 4):
            self.spmv_is_right(k)
        assert self.dev.get_status() == 0


@pytest.mark.parametrize("in_graph", [(), (1,), (4,), (1, 4)])
def test_reads_after_replays(dcsr, in_graph):
    """A graph of an update, alone or with SpMVs of one or four right-hand
    sides behind it; everything read after each run."""
    q = Case(dcsr, 1 + len(in_graph))
    q.triples()
    q.update()  # (sizes the scratch)
    torch.cuda.synchronize()
    q.all_right("before")
    g = q.captured(q.update, *[lambda k=k: q.spmv(k) for k in in_graph])
    q.all_right("captured, not run")
    for it in range(3):
        q.run(g)
        if in_graph:
            k = in_graph[-1]
            for j in range(k):
                np.testing.assert_allclose(q.y[:, j].cpu().numpy(), q.orc.spmv(q.x[:, j].cpu().numpy().copy()), rtol=0,
                                           atol=1e-9)
        q.all_right(f"run {it}")


def test_stale_tables_at_the_capture(dcsr):
    """Tables stale before the capture, built in it, read before its first run."""
    q = Case(dcsr, 7)
    q.spmv(1)
    q.spmv(4)
    q.triples()
    q.update()
    g = q.captured(q.update, lambda: q.spmv(1), lambda: q.spmv(4))
    q.all_right("captured, not run")
    q.run(g)
    q.all_right("run")


def test_two_graphs(dcsr):
    """Updates in two captures, tables built in one of them only."""
    q = Case(dcsr, 8)
    q.triples()
    q.update()
    q.spmv(4)
    q.spmv(1)
    torch.cuda.synchronize()
    g1 = q.captured(q.update)
    g2 = q.captured(q.update, lambda: q.spmv(1))
    for it in range(2):
        q.run(g2)
        q.all_right(f"g2 {it}")
        q.run(g1)
        q.all_right(f"g1 {it}")


@pytest.mark.parametrize("read", ["spmv", "sum", "csr"])
def test_prepared_by_calls_before(dcsr, read):
    """A load, one call of each kind, then the capture: an update of less than a
    scan block, and a read whose tables the graph has to build."""
    q = Case(dcsr, 9)
    L, s = dcsr.lib(), q.s.cuda_stream
    room = q.dev.nnz() + 10 * q.T
    rp, ec, ev = (torch.zeros(N + 1, dtype=torch.int32).cuda(), torch.zeros(room, dtype=torch.int32).cuda(),
                  torch.zeros(room, dtype=torch.float64).cuda())
    call = {
        "spmv": lambda: q.spmv(1),
        "sum": lambda: q.check(L.dcsr_row_reduce(q.dev.h, dcsr.REDUCE_SUM, q.y.data_ptr(), s)),
        "csr": lambda: q.check(L.dcsr_to_csr(q.dev.h, rp.data_ptr(), ec.data_ptr(), ev.data_ptr(), s)),
    }[read]
    call()
    q.triples()
    q.update()
    g = q.captured(q.update, call)
    for it in range(2):
        q.run(g)
        if read == "csr":
            rp_o, c_o, v_o = q.orc.export_csr()
            np.testing.assert_array_equal(rp.cpu().numpy(), rp_o)
            np.testing.assert_array_equal(ec.cpu().numpy()[: c_o.size], c_o)
            np.testing.assert_array_equal(ev.cpu().numpy()[: c_o.size], v_o)
        q.all_right(f"run {it}")


def test_never_loaded(dcsr):
    """A matrix of updates alone; the call before the capture has four right-hand
    sides, the one in it has one."""
    q = Case(dcsr, 10, load=False)
    for _ in range(3):
        q.triples()
        q.update()
    q.spmv(4)
    g = q.captured(lambda: q.spmv(1), q.update, lambda: q.spmv(1))
    q.all_right("captured, not run")
    q.run(g)
    np.testing.assert_allclose(q.y[:, 0].cpu().numpy(), q.orc.spmv(q.x[:, 0].cpu().numpy().copy()), rtol=0, atol=1e-9)
    q.all_right("run")
