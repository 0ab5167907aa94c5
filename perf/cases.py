"""The work that a user of the library has it do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes what a program holds on the
GPU before a call (matrices, triples, right-hand sides, a captured batch, a
server), ``run`` is one pass through the public entry points, ``exact`` the
same results in 64 bits from plain torch.  All inputs are seeded synthetic
data of the shapes and value distributions of ``dcsr_b200.workloads``.

What a case does is its ``op``:

* ``spmv``    y = alpha*A@x + beta*y on a matrix that has had an update
* ``round``   a load from CSR, then update rounds, each followed by an SpMV,
              the row sums and the export to CSR
* ``load``    a load from unsorted COO triples, and the export to CSR
* ``spgemm``  C = A*A into a kept handle, and C's export to CSR
* ``batch``   one launch of a captured batch: an update and an SpMV on each of
              many matrices of uneven size, and the statuses
* ``served``  a burst of update, SpMV and export requests to a server, until
              every result is there
"""
from __future__ import annotations

import math

import torch

from dcsr_b200 import api

DTYPES = {"f32": torch.float32, "f64": torch.float64}
BYTES = {"f32": 4, "f64": 8}
# entries of the largest matrix: 2^20 rows of mean degree 16
MOST_ENTRIES = 1 << 24
RMAT = (0.57, 0.19, 0.19, 0.05)


def listed():
    return [
        # one SpMV of a small matrix: an iterative caller's inner step, where
        # the launches count
        dict(name="spmv_small", op="spmv", graph="poisson", rows=4096, cols=4096, degree=12, dtype="f32", k=1,
             alpha=1.0, beta=0.0, triples=8192),
        # the SpMV of the power-law update stream: rows from empty to tens of
        # thousands of entries, some of them in several segments
        dict(name="spmv_rmat", op="spmv", graph="rmat", rows=1 << 20, cols=1 << 20, degree=16, dtype="f32", k=1,
             alpha=1.0, beta=0.0, triples=1 << 20),
        # a block of right-hand sides on one of the batched form's larger matrices
        dict(name="spmv_rhs8", op="spmv", graph="poisson", rows=200_003, cols=200_003, degree=40, dtype="f32", k=8,
             alpha=1.0, beta=0.0, triples=50_001),
        # double precision, an odd number of right-hand sides, rectangular, accumulating
        dict(name="spmv_rhs3_f64", op="spmv", graph="poisson", rows=100_003, cols=65_537, degree=20, dtype="f64", k=3,
             alpha=1.5, beta=0.5, triples=20_011),
        # the small plain workload: 4 rounds of 8192 triples (merged) on 4096 rows
        dict(name="round_small", op="round", graph="poisson", rows=4096, cols=4096, degree=12, dtype="f32", mode=0,
             rounds=4, triples=8192),
        # a mid-size double-precision matrix in append mode, odd sizes
        dict(name="round_append_f64", op="round", graph="poisson", rows=50_021, cols=50_021, degree=14, dtype="f64",
             mode=1, rounds=2, triples=100_003),
        # the power-law update stream: rounds of 1M skewed triples
        dict(name="round_rmat", op="round", graph="rmat", rows=1 << 20, cols=1 << 20, degree=16, dtype="f32", mode=0,
             rounds=2, triples=1 << 20),
        # 16.8M unsorted triples of the same graph, duplicates summed
        dict(name="load_rmat", op="load", graph="rmat", rows=1 << 20, cols=1 << 20, degree=16, dtype="f32", mode=0),
        # the double-precision banded product
        dict(name="spgemm_banded", op="spgemm", rows=1 << 17, band=2, off=8, dtype="f64"),
        # a product of rows with several hundred products each
        dict(name="spgemm_wide", op="spgemm", rows=20_011, band=2, off=24, dtype="f32"),
        # the batched form: an update and an SpMV on each matrix, one graph launch
        dict(name="batch_48", op="batch", count=48, min_rows=1000, max_rows=128_000, min_triples=100,
             max_triples=50_000, dtype="f32"),
        # the served form: a burst of mixed requests over resident matrices
        dict(name="served_64", op="served", count=24, min_rows=1000, max_rows=128_000, min_triples=10,
             max_triples=50_000, requests=64, dtype="f32"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _graph(rng):
    """A power-law or a Poisson matrix of the listed ones' range."""
    if rng.random() < 0.4:
        scale = rng.randint(12, 20)
        degree = rng.randint(4, 16)
        return dict(graph="rmat", rows=1 << scale, cols=1 << scale, degree=degree)
    rows = _log_uniform(rng, 1000, 262_144)
    cols = rows if rng.random() < 0.7 else _log_uniform(rng, 1000, 262_144)
    return dict(graph="poisson", rows=rows, cols=cols, degree=rng.randint(4, min(64, MOST_ENTRIES // rows)))


def draw(rng):
    op = rng.choice(["spmv", "spmv", "round", "round", "load", "spgemm", "batch", "served"])
    dtype = rng.choice(["f32", "f32", "f64"])
    if op == "spmv":
        g = _graph(rng)
        if g["rows"] * g["degree"] > MOST_ENTRIES // 2:
            k = rng.choice([1, 2])
        else:
            k = rng.randint(1, 8)
        accumulate = rng.random() < 0.3
        return dict(op=op, **g, dtype=dtype, k=k, alpha=1.5 if accumulate else 1.0, beta=0.5 if accumulate else 0.0,
                    triples=_log_uniform(rng, 10, 1 << 20))
    if op == "round":
        g = _graph(rng)
        return dict(op=op, **g, dtype="f32" if g["rows"] > 1 << 19 else dtype, mode=rng.choice([0, 0, 1]),
                    rounds=rng.randint(1, 2 if g["rows"] > 1 << 17 else 4),
                    triples=_log_uniform(rng, 10, 1 << 20 if g["rows"] > 1 << 17 else 1 << 17))
    if op == "load":
        g = _graph(rng)
        return dict(op=op, **g, dtype="f32" if g["rows"] > 1 << 19 else dtype, mode=rng.choice([0, 0, 1]))
    if op == "spgemm":
        off = rng.randint(3, 24)
        most = min(1 << 17, 22_000_000 // (5 + off) ** 2)
        return dict(op=op, rows=_log_uniform(rng, 1000, most), band=2, off=off, dtype=dtype)
    sizes = dict(min_rows=1000, max_rows=_log_uniform(rng, 4000, 128_000),
                 max_triples=_log_uniform(rng, 1000, 50_000), dtype="f32")
    if op == "batch":
        return dict(op=op, count=rng.randint(8, 48), min_triples=100, **sizes)
    return dict(op=op, count=rng.randint(8, 24), min_triples=10, requests=rng.randint(24, 64), **sizes)


# ------------------------------------------------------------------ inputs

DEV = "cuda"


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1_000_003 + salt)
    return g


def _values(case, n, g):
    """U(0,1) on the power-law graph, else U(-1,1)."""
    v = torch.rand(n, device=DEV, dtype=DTYPES[case["dtype"]], generator=g)
    return v if case.get("graph") == "rmat" else v * 2 - 1


def _poisson(rows, cols, degree, g):
    """rows * degree entries in uniform rows and columns: Poisson row lengths
    whose sum does not depend on the seed."""
    r = torch.sort(torch.randint(0, rows, (rows * degree,), device=DEV, dtype=torch.int32, generator=g))[0]
    return r, torch.randint(0, cols, (r.numel(),), device=DEV, dtype=torch.int32, generator=g)


def _rmat(rows, degree, g):
    a, b, c, _ = RMAT
    n = rows * degree
    r = torch.zeros(n, device=DEV, dtype=torch.int32)
    k = torch.zeros(n, device=DEV, dtype=torch.int32)
    for level in range(rows.bit_length() - 1):
        u = torch.rand(n, device=DEV, generator=g)
        r |= (u >= a + b).to(torch.int32) << level
        k |= (((u >= a) & (u < a + b)) | (u >= a + b + c)).to(torch.int32) << level
    return r, k


def _triples(case, base_rows, count, g):
    """An update batch: on the power-law graph rows in proportion to their
    length, else uniform rows; uniform columns; about half of them on columns
    of existing entries in a Poisson matrix's case."""
    r, c = base_rows
    if case["graph"] == "rmat":
        pick = torch.randint(0, r.numel(), (count,), device=DEV, generator=g)
        ur = r[pick]
        uc = torch.randint(0, case["cols"], (count,), device=DEV, dtype=torch.int32, generator=g)
    else:
        pick = torch.randint(0, r.numel(), (count,), device=DEV, generator=g)
        half = torch.rand(count, device=DEV, generator=g) < 0.5
        ur = torch.where(half, r[pick],
                         torch.randint(0, case["rows"], (count,), device=DEV, dtype=torch.int32, generator=g))
        uc = torch.where(half, c[pick],
                         torch.randint(0, case["cols"], (count,), device=DEV, dtype=torch.int32, generator=g))
    return ur, uc, _values(case, count, g)


def _edges(case, seed):
    g = _gen(seed)
    if case["graph"] == "rmat":
        r, c = _rmat(case["rows"], case["degree"], g)
    else:
        r, c = _poisson(case["rows"], case["cols"], case["degree"], g)
    return r, c, _values(case, r.numel(), g), g


def _banded(case, seed):
    """Band of half-width `band` plus `off` uniform columns in every row, N(0,1)."""
    g = _gen(seed)
    n, w = case["rows"], case["band"]
    i = torch.arange(n, device=DEV, dtype=torch.int64)
    band = i[:, None] + torch.arange(-w, w + 1, device=DEV)[None, :]
    off = torch.randint(0, n, (n, case["off"]), device=DEV, generator=g)
    c = torch.cat([band, off], 1)
    r = i[:, None].expand_as(c)
    ok = (c >= 0) & (c < n)
    r, c = r[ok].to(torch.int32), c[ok].to(torch.int32)
    v = torch.randn(r.numel(), device=DEV, dtype=DTYPES[case["dtype"]], generator=g)
    return r, c, v


def _members(case, seed):
    """The matrices of a batch or a server: sizes from the case alone (so
    passes of different seeds do the same work), contents from the seed."""
    import random
    rng = random.Random(case["count"] * 7919 + case["max_rows"])
    out = []
    for i in range(case["count"]):
        n = _log_uniform(rng, case["min_rows"], case["max_rows"])
        m = dict(graph="poisson", rows=n, cols=n, degree=rng.randint(4, 64), dtype=case["dtype"],
                 triples=_log_uniform(rng, case["min_triples"], case["max_triples"]), k=rng.choice([1, 2, 4, 8]))
        m["seed"] = seed * 1009 + i
        out.append(m)
    return out


def _burst(case):
    """The request mix: 40% updates, 50% SpMVs with 1 to 8 right-hand sides,
    10% exports, over uniform matrices."""
    import random
    rng = random.Random(case["requests"] * 104_729 + case["count"])
    out = []
    for _ in range(case["requests"]):
        u, i = rng.random(), rng.randrange(case["count"])
        if u < 0.4:
            out.append(("update", i, _log_uniform(rng, case["min_triples"], case["max_triples"])))
        elif u < 0.9:
            out.append(("spmv", i, rng.randint(1, 8)))
        else:
            out.append(("export", i, 0))
    return out


def _rhs(n, k, dtype, g):
    x = torch.rand((n, k) if k > 1 else (n,), device=DEV, dtype=DTYPES[dtype], generator=g)
    return x * 2 - 1


# ----------------------------------------------------------------- prepare

class State:
    """What a program holds between calls."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _csr_room(rows, entries, dtype):
    """Export buffers for at most that many entries, zero past the matrix's own."""
    return dict(row_ptr=torch.zeros(rows + 1, device=DEV, dtype=torch.int32),
                cols=torch.zeros(entries, device=DEV, dtype=torch.int32),
                vals=torch.zeros(entries, device=DEV, dtype=DTYPES[dtype]))


def _export(A, out):
    """A as CSR in the caller's buffers, through the C ABI: their entries, then the arrays."""
    assert A.nnz() <= out["cols"].numel()
    status = api.lib().dcsr_to_csr(A.h, out["row_ptr"].data_ptr(), out["cols"].data_ptr(), out["vals"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
    assert status == api.OK
    return out


def _padded(v, entries):
    return torch.cat([v, torch.zeros(entries - v.numel(), device=DEV, dtype=v.dtype)])


def prepare(case, seed):
    return globals()["_prepare_" + case["op"]](case, seed)


def _spmv_inputs(case, seed):
    r, c, v, g = _edges(case, seed)
    u = _triples(case, (r, c), case["triples"], g)
    x = _rhs(case["cols"], case["k"], case["dtype"], g)
    y = _rhs(case["rows"], case["k"], case["dtype"], g)
    return (r, c, v), u, x, y


def _prepare_spmv(case, seed):
    (r, c, v), u, x, y = _spmv_inputs(case, seed)
    A = api.DcsrMatrix(case["rows"], case["cols"], DTYPES[case["dtype"]])
    A.from_coo(r, c, v)
    assert A.update(*u) == api.OK
    A.bin_rows()
    return State(op="spmv", A=A, x=x, y=y, alpha=case["alpha"], beta=case["beta"])


def _round_inputs(case, seed):
    r, c, v, g = _edges(case, seed)
    batches = [_triples(case, (r, c), case["triples"], g) for _ in range(case["rounds"])]
    x = _rhs(case["cols"], 1, case["dtype"], g)
    key, order = torch.sort(r.to(torch.int64) * case["cols"] + c, stable=True)
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]
    return key[first], v[order][first], batches, x


def _prepare_round(case, seed):
    key, v, batches, x = _round_inputs(case, seed)
    rows = torch.div(key, case["cols"], rounding_mode="floor")
    row_ptr = torch.zeros(case["rows"] + 1, device=DEV, dtype=torch.int32)
    row_ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=case["rows"]), 0)
    cols = (key % case["cols"]).to(torch.int32)
    A = api.DcsrMatrix(case["rows"], case["cols"], DTYPES[case["dtype"]], mode=case["mode"])
    room = _entries(case) + case["rounds"] * case["triples"]
    out = [dict(_csr_room(case["rows"], room, case["dtype"]),
                y=torch.zeros(case["rows"], device=DEV, dtype=DTYPES[case["dtype"]]),
                sums=torch.zeros(case["rows"], device=DEV, dtype=DTYPES[case["dtype"]])) for _ in batches]
    return State(op="round", A=A, csr=(row_ptr, cols, v), batches=batches, x=x, out=out)


def _prepare_load(case, seed):
    r, c, v, _ = _edges(case, seed)
    order = torch.randperm(r.numel(), device=DEV, generator=_gen(seed, 1))
    A = api.DcsrMatrix(case["rows"], case["cols"], DTYPES[case["dtype"]], mode=case["mode"])
    return State(op="load", A=A, coo=(r[order], c[order], v[order]),
                 out=_csr_room(case["rows"], _entries(case), case["dtype"]))


def _prepare_spgemm(case, seed):
    r, c, v = _banded(case, seed)
    A = api.DcsrMatrix(case["rows"], case["rows"], DTYPES[case["dtype"]])
    A.from_coo(r, c, v)
    C = api.DcsrMatrix(case["rows"], case["rows"], DTYPES[case["dtype"]])
    room = case["rows"] * (2 * case["band"] + 1 + case["off"]) ** 2
    return State(op="spgemm", A=A, C=C, out=_csr_room(case["rows"], room, case["dtype"]))


def _member_inputs(m):
    r, c, v, g = _edges(m, m["seed"])
    u = _triples(m, (r, c), m["triples"], g)
    return (r, c, v), u, _rhs(m["cols"], m["k"], m["dtype"], g), g


def _prepare_batch(case, seed):
    mats, work = [], []
    members = _members(case, seed)
    y = torch.zeros(sum(m["rows"] * m["k"] for m in members), device=DEV, dtype=DTYPES[case["dtype"]])
    at = 0
    for m in members:
        coo, u, x, _ = _member_inputs(m)
        A = api.DcsrMatrix(m["rows"], m["cols"], DTYPES[m["dtype"]])
        A.from_coo(*coo)
        n = m["rows"] * m["k"]
        work.append(dict(matrix=A, rows=u[0], cols=u[1], vals=u[2], x=x, y=y[at:at + n].view(x.shape)))
        at += n
        mats.append(A)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        batch = api.DcsrBatch(work)
        batch.capture()
    stream.synchronize()
    return State(op="batch", mats=mats, batch=batch, stream=stream, y=y)


def _served_inputs(case, seed):
    """Per request its tensors: triples, or a right-hand side."""
    members = _members(case, seed)
    coos = [_member_inputs(m)[0] for m in members]
    g = _gen(seed, 2)
    reqs = []
    for kind, i, size in _burst(case):
        m = members[i]
        if kind == "update":
            reqs.append((kind, i, _triples(m, coos[i][:2], size, g)))
        elif kind == "spmv":
            reqs.append((kind, i, _rhs(m["cols"], size, case["dtype"], g)))
        else:
            reqs.append((kind, i, None))
    return members, coos, reqs


def _export_room(members, coos, reqs):
    """Per export its place in the export buffers: entries the matrix can hold."""
    room = [c[0].numel() for c in coos]
    for kind, i, t in reqs:
        if kind == "update":
            room[i] += t[0].numel()
    return [room[i] if kind == "export" else 0 for kind, i, _ in reqs]


def _prepare_served(case, seed):
    members, coos, reqs = _served_inputs(case, seed)
    dt = DTYPES[case["dtype"]]
    mats = []
    for m, coo in zip(members, coos):
        A = api.DcsrMatrix(m["rows"], m["cols"], dt)
        A.from_coo(*coo)
        mats.append(A)
    room = _export_room(members, coos, reqs)
    ny = sum(members[i]["rows"] * (1 if t.dim() == 1 else t.shape[1]) for kind, i, t in reqs if kind == "spmv")
    nr = sum(members[i]["rows"] + 1 for kind, i, _ in reqs if kind == "export")
    y = torch.zeros(ny, device=DEV, dtype=dt)
    rp = torch.zeros(nr, device=DEV, dtype=torch.int32)
    oc = torch.zeros(sum(room), device=DEV, dtype=torch.int32)
    ov = torch.zeros(sum(room), device=DEV, dtype=dt)
    calls, aty, atr, ate = [], 0, 0, 0
    for (kind, i, t), n in zip(reqs, room):
        rows = members[i]["rows"]
        if kind == "update":
            calls.append((kind, (i,) + tuple(t)))
        elif kind == "spmv":
            k = 1 if t.dim() == 1 else t.shape[1]
            calls.append((kind, (i, t, y[aty:aty + rows * k].view((rows,) if k == 1 else (rows, k)))))
            aty += rows * k
        else:
            calls.append((kind, (i, rp[atr:atr + rows + 1], oc[ate:ate + n], ov[ate:ate + n])))
            atr += rows + 1
            ate += n
    torch.cuda.synchronize()
    server = api.DcsrServer(mats, depth=8, mem_budget=8 << 30, workers=4)
    return State(op="served", mats=mats, server=server, calls=calls, y=y, row_ptr=rp, cols=oc, vals=ov)


# --------------------------------------------------------------------- run

def run(state):
    return globals()["_run_" + state.op](state)


def _run_spmv(s):
    return s.A.spmv(s.x, s.y, alpha=s.alpha, beta=s.beta)


def _run_round(s):
    s.A.from_csr(*s.csr)
    for batch, out in zip(s.batches, s.out):
        out["status"] = s.A.update(*batch)
        s.A.spmv(s.x, out["y"])
        s.A.row_reduce(api.REDUCE_SUM, out["sums"])
        _export(s.A, out)
    return s.out


def _run_load(s):
    s.A.from_coo(*s.coo)
    return _export(s.A, s.out)


def _run_spgemm(s):
    s.A.spgemm(s.A, s.C)
    return _export(s.C, s.out)


def _run_batch(s):
    with torch.cuda.stream(s.stream):
        s.batch.launch()
        status = s.batch.status()
        if status.any():
            s.batch.repair(status)
    return dict(y=s.y, status=status)


def _run_served(s):
    submit = dict(update=s.server.submit_update, spmv=s.server.submit_spmv, export=s.server.submit_export)
    tickets = [submit[kind](*args) for kind, args in s.calls]
    results = [s.server.wait(t) for t in tickets]
    return dict(y=s.y, row_ptr=s.row_ptr, cols=s.cols, vals=s.vals,
                status=torch.tensor([r["status"] for r in results]))


# -------------------------------------------------------------------- work

def _entries(case):
    return case["rows"] * case["degree"]


def work(case):
    sv = BYTES[case["dtype"]] if "dtype" in case else 4
    if case["op"] == "spmv":
        e = _entries(case) + case["triples"]
        nbytes = e * (4 + sv) + 12 * case["rows"] + case["k"] * sv * (
            case["rows"] * (2 if case["beta"] else 1) + case["cols"])
        return {"bytes": nbytes, "flops": 2 * e * case["k"]}
    if case["op"] == "round":
        e, t, n = _entries(case), case["triples"], case["rounds"]
        nbytes = e * (4 + sv) + 4 * case["rows"]
        flops = 0
        for i in range(1, n + 1):
            nbytes += t * (8 + sv) + sv * case["cols"] + (4 + 2 * sv) * case["rows"] + (e + i * t) * (4 + sv)
            flops += t + 3 * (e + i * t)
        return {"bytes": nbytes, "flops": flops}
    if case["op"] == "load":
        e = _entries(case)
        return {"bytes": e * (8 + sv) + e * (4 + sv) + 4 * case["rows"], "flops": e}
    if case["op"] == "spgemm":
        n, d = case["rows"], 2 * case["band"] + 1 + case["off"]
        products = n * d * d
        return {"bytes": n * d * (4 + sv) + 4 * n + products * (4 + sv) + 4 * n, "flops": 2 * products}
    nbytes = flops = 0
    members = _members(case, 0)
    if case["op"] == "batch":
        for m in members:
            e = _entries(m) + m["triples"]
            nbytes += e * (4 + sv) + m["triples"] * (8 + sv) + 2 * m["k"] * sv * m["rows"] + 12 * m["rows"]
            flops += 2 * e * m["k"] + m["triples"]
        return {"bytes": nbytes, "flops": flops}
    for kind, i, size in _burst(case):
        m = members[i]
        e = _entries(m)
        if kind == "update":
            nbytes += size * (8 + sv) + size * (4 + sv)
            flops += size
        elif kind == "spmv":
            nbytes += e * (4 + sv) + 2 * size * sv * m["rows"] + 12 * m["rows"]
            flops += 2 * e * size
        else:
            nbytes += 2 * e * (4 + sv) + 16 * m["rows"]
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------- exact

def _coalesce(r, c, v, cols):
    """Sorted unique (row, column) keys and their sums in 64 bits."""
    key, where = torch.unique(r.to(torch.int64) * cols + c, return_inverse=True)
    return key, torch.zeros(key.numel(), device=DEV, dtype=torch.float64).index_add_(0, where, v.double())


def _product(r, c, v, x, rows):
    """A @ x in 64 bits for a matrix given by its triples."""
    x = x.double()
    out = torch.zeros((rows,) + tuple(x.shape[1:]), device=DEV, dtype=torch.float64)
    step = max(1, (1 << 26) // max(1, x[:1].numel()))
    for a in range(0, r.numel(), step):
        xv = x[c[a:a + step].long()]
        p = v[a:a + step].double()
        out.index_add_(0, r[a:a + step].long(), xv * (p[:, None] if x.dim() > 1 else p))
    return out


def _join(coo, u):
    return tuple(torch.cat([a, b]) for a, b in zip(coo, u))


def exact(case, seed):
    return globals()["_exact_" + case["op"]](case, seed)


def _exact_spmv(case, seed):
    coo, u, x, y = _spmv_inputs(case, seed)
    p = _product(*_join(coo, u), x, case["rows"]) * case["alpha"]
    return p + case["beta"] * y.double() if case["beta"] else p


def _exact_round(case, seed):
    key, v, batches, x = _round_inputs(case, seed)
    r = torch.div(key, case["cols"], rounding_mode="floor").to(torch.int32)
    coo = (r, (key % case["cols"]).to(torch.int32), v)
    out = []
    for u in batches:
        coo = _join(coo, u)
        y = _product(*coo, x, case["rows"])
        sums = torch.zeros(case["rows"], device=DEV, dtype=torch.float64).index_add_(0, coo[0].long(), coo[2].double())
        if case["mode"] == api.MERGE:
            vals = _coalesce(*coo, case["cols"])[1]
        else:
            vals = coo[2][torch.sort(coo[0], stable=True)[1]].double()
        vals = _padded(vals, _entries(case) + case["rounds"] * case["triples"])
        out.append(dict(status=None, y=y, sums=sums, row_ptr=None, cols=None, vals=vals))
    return out


def _exact_load(case, seed):
    r, c, v, _ = _edges(case, seed)
    order = torch.randperm(r.numel(), device=DEV, generator=_gen(seed, 1))
    r, c, v = r[order], c[order], v[order]
    if case["mode"] == api.MERGE:
        vals = _coalesce(r, c, v, case["cols"])[1]
    else:
        vals = v[torch.sort(r, stable=True)[1]].double()
    return dict(row_ptr=None, cols=None, vals=_padded(vals, _entries(case)))


def _exact_spgemm(case, seed):
    n = case["rows"]
    key, v = _coalesce(*_banded(case, seed), n)
    v = v.to(DTYPES[case["dtype"]]).double()
    r, c = torch.div(key, n, rounding_mode="floor"), key % n
    lens = torch.bincount(r, minlength=n)
    start = torch.cumsum(lens, 0) - lens
    reps = lens[c]
    at = torch.repeat_interleave(torch.arange(r.numel(), device=DEV), reps)
    within = torch.arange(at.numel(), device=DEV) - torch.repeat_interleave(torch.cumsum(reps, 0) - reps, reps)
    b = start[c[at]] + within
    return dict(row_ptr=None, cols=None, vals=_padded(_coalesce(r[at], c[b], v[at] * v[b], n)[1],
                                                       n * (2 * case["band"] + 1 + case["off"]) ** 2))


def _exact_batch(case, seed):
    ys = []
    for m in _members(case, seed):
        coo, u, x, _ = _member_inputs(m)
        ys.append(_product(*_join(coo, u), x, m["rows"]).reshape(-1))
    return dict(y=torch.cat(ys), status=None)


def _exact_served(case, seed):
    members, coos, reqs = _served_inputs(case, seed)
    room = _export_room(members, coos, reqs)
    coos = list(coos)
    ys, vals = [torch.zeros(0, device=DEV, dtype=torch.float64)], [torch.zeros(0, device=DEV, dtype=torch.float64)]
    for (kind, i, t), n in zip(reqs, room):
        if kind == "update":
            coos[i] = _join(coos[i], t)
        elif kind == "spmv":
            ys.append(_product(*coos[i], t, members[i]["rows"]).reshape(-1))
        else:
            vals.append(_padded(_coalesce(*coos[i], members[i]["cols"])[1], n))
    return dict(y=torch.cat(ys), row_ptr=None, cols=None, vals=torch.cat(vals), status=None)
