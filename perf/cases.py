"""The products that are timed: what programs built on this library ask of it.

A case is a dict of plain values: the entry point (`call`), the sparse matrix
(`matrix`, `rows`, `degree`), the dense width `n`, and the options of the
call.  Matrices are square.  `matrix` is one of

  uniform   exactly `degree` uniformly random columns per row
  random    Poisson(`degree`) uniformly random columns per row: rows of unequal
            length, some of them empty
  powerlaw  out-degrees p(k) ~ (k + 0.16)^-2.1 on [1, 4096] scaled to an average
            of `degree`, columns by preferential attachment

The ranges: 1k to 1M rows, 2 to 32 nonzeros per row on average, 1 to 512 dense
columns, both dense layouts, every storage format of the mixed-precision call,
batches and servers of matrices of 1k to 64k rows.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "da-spmmul-kernel_b200"))

import daspmm as D  # noqa: E402

ALGS = {"csr_scalar": 0, "csr_vector": 1, "coo_scalar": 2, "coo_vector": 3, "balanced": 4}
FORMATS = {"f32": 0, "bf16": 1, "f16": 2, "e4m3": 3}
TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SERVE_WIDTHS = (16, 64, 256)
MOST = 2_200_000_000  # nonzeros times dense columns of the largest case


def listed():
    return [
        # the small uniform matrix of the benchmark: a call that is all launch latency
        dict(name="uniform_4k_n32", call="spmm", alg="balanced", layout="row", matrix="uniform",
             rows=4096, degree=16, n=32, beta=0.0),
        # the benchmark's headline: one power-law graph, 128 features
        dict(name="powerlaw_262k_n128", call="spmm", alg="balanced", layout="row",
             matrix="powerlaw", rows=262144, degree=4.74, n=128, beta=0.0),
        # a sparse matrix times one vector: the inner step of an iterative solver
        dict(name="spmv_262k", call="spmm", alg="balanced", layout="row", matrix="random",
             rows=262144, degree=12, n=1, beta=0.0),
        # a sparse graph with rows that hold nothing, 64 features
        dict(name="empty_rows_400k_n64", call="spmm", alg="balanced", layout="row",
             matrix="random", rows=400000, degree=3, n=64, beta=0.0),
        # a width that no vector load divides (a class count), added to what C holds
        dict(name="ragged_150k_n41_add", call="spmm", alg="balanced", layout="row",
             matrix="powerlaw", rows=150001, degree=8, n=41, beta=1.0),
        # the dispatcher of the reference called as its own driver does: COO, row-major
        dict(name="compat_coo_262k_n32", call="compat", alg="coo_scalar", layout="row",
             matrix="powerlaw", rows=262144, degree=4.74, n=32),
        # the same dispatcher, column-major operands, CSR
        dict(name="compat_csr_col_100k_n16", call="compat", alg="csr_vector", layout="col",
             matrix="random", rows=100000, degree=8, n=16),
        # operands of a column-major program (Fortran, BLAS conventions)
        dict(name="colmajor_262k_n128", call="spmm", alg="balanced", layout="col",
             matrix="powerlaw", rows=262144, degree=4.74, n=128, beta=0.0),
        # activations quantised to E4M3 on the way in, then the product
        dict(name="e4m3_262k_n256", call="mixed", val="bf16", b="e4m3", quantize=True,
             matrix="random", rows=262144, degree=8, n=256, beta=0.0),
        # many graphs of uneven sizes in one launch (mini-batches of subgraphs)
        dict(name="batch_48_n64", call="batch", val="f32", b="bf16", instances=48, n=64),
        # a burst of requests to a server with resident matrices, waited for
        dict(name="serve_24", call="serve", matrices=8, requests=24),
        # one large matrix kept as a plan, many products, wide features
        dict(name="plan_1m_n256", call="plan", matrix="random", rows=1048576, degree=8, n=256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choice(["spmm"] * 5 + ["compat"] * 3 + ["mixed"] * 2 + ["batch", "serve", "plan"])
    if call == "batch":
        val, b = rng.choice([("f32", "f32"), ("f32", "bf16"), ("bf16", "bf16"), ("bf16", "e4m3")])
        return dict(call=call, val=val, b=b, instances=rng.randint(8, 56),
                    n=rng.choice([32, 64, 96, 128]))
    if call == "serve":
        return dict(call=call, matrices=rng.randint(4, 12), requests=rng.randint(8, 48))
    c = dict(call=call, matrix=rng.choice(["uniform", "random", "powerlaw"]),
             degree=round(_log(rng, 2, 32)))
    # an ordinary width, any width, or one of the reference's powers of two
    kind = rng.random()
    if call == "mixed":
        n = 32 * rng.randint(1, 16)
        val, b = rng.choice([("bf16", "bf16"), ("f16", "f16"), ("f32", "e4m3"), ("bf16", "e4m3")])
        c.update(val=val, b=b, quantize=rng.random() < 0.5, beta=rng.choice([0.0, 0.0, 0.5]))
    elif call == "compat":
        n = 2 ** rng.randint(0, 7)
        c.update(alg=rng.choice(["csr_scalar", "csr_vector", "coo_scalar", "coo_vector"]),
                 layout=rng.choice(["row", "col"]))
    else:
        n = (2 ** rng.randint(5, 9) if kind < 0.4 else 4 * rng.randint(1, 64) if kind < 0.7
             else round(_log(rng, 1, 512)))
        if call == "spmm":
            c.update(alg="balanced", layout=rng.choice(["row", "row", "row", "col"]),
                     beta=rng.choice([0.0, 0.0, 0.5, 1.0]))
    c["n"] = n
    most = min(1_048_576, int(MOST / (n * c["degree"])))
    c["rows"] = min(most, round(_log(rng, 1000, 1_048_576)))
    return c


# ------------------------------------------------------------------ inputs
def _degrees(kind, rows, degree, g):
    if kind == "uniform":
        return torch.full((rows,), int(degree), device="cuda")
    if kind == "random":
        return torch.poisson(torch.full((rows,), float(degree), device="cuda"), generator=g).long()
    k = torch.arange(1, min(4096, rows) + 1, device="cuda", dtype=torch.float64)
    p = (k + 0.16) ** -2.1
    p /= p.sum()
    cdf = p.cumsum(0)
    u = torch.rand(rows, generator=g, device="cuda", dtype=torch.float64)
    d = k[torch.searchsorted(cdf, u).clamp_(max=k.numel() - 1)]
    return (d * (degree / float((k * p).sum()))).round_().long().clamp_(1, k.numel())


def _csr(kind, rows, degree, seed):
    """(rowPtr, colIdx, values) on the GPU: columns sorted and distinct in each row."""
    g = torch.Generator("cuda").manual_seed(seed)
    deg = _degrees(kind, rows, degree, g)
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), deg)
    nnz = row.numel()
    if kind == "powerlaw":
        # an entry takes a new column, or the column of an entry before it
        at = torch.arange(nnz, device="cuda")
        j = (torch.rand(nnz, generator=g, device="cuda", dtype=torch.float64) * (rows + at)).long()
        src = torch.where(j < rows, at, j - rows)
        while True:
            nxt = src[src]
            if torch.equal(nxt, src):
                break
            src = nxt
        col = j[src]
    else:
        col = torch.randint(rows, (nnz,), generator=g, device="cuda")
    key = torch.unique(row * rows + col)
    row, col = key // rows, key % rows
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.bincount(row, minlength=rows).cumsum(0)
    val = torch.rand(key.numel(), generator=g, device="cuda") * 2 - 1
    return ptr.int(), col.int(), val


def _matrix(kind, rows, degree, seed):
    ptr, col, val = _csr(kind, rows, degree, seed)
    return D.DeviceCsr(D.Csr(rows, rows, ptr.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()))


def _dense(rows, n, seed, fmt="f32"):
    g = torch.Generator("cuda").manual_seed(seed)
    return (torch.rand(rows, n, generator=g, device="cuda") * 2 - 1).to(TORCH[fmt])


def _to_e4m3(x):
    """(codes, per-column scales) of a float32 matrix in E4M3, by torch alone."""
    top = x.abs().amax(0)
    scale = torch.where(top > 0, top / torch.full_like(top, 448.0), torch.ones_like(top))
    return (x / scale).to(torch.float8_e4m3fn), scale


def _operands(c, seed):
    """(C to add to, B) of a single product, in the layout of the call."""
    shape = (c["rows"], c["n"]) if c.get("layout", "row") == "row" else (c["n"], c["rows"])
    adds = c.get("beta", 0.0) != 0.0 or c.get("alg", "").startswith("coo")
    C = _dense(*shape, seed + 2) if adds else torch.empty(shape, device="cuda")
    return C, _dense(*shape, seed + 1)


def _instances(c, seed):
    """(kind, rows, degree, seed) of each matrix of a batch or a server; the sizes are the case's own."""
    count = c.get("instances") or c["matrices"]
    r = torch.rand(count, 2, generator=torch.Generator().manual_seed(count))
    out = []
    for i, (u, v) in enumerate(r.tolist()):
        rows = int(1000 * 65.536 ** u)
        if c["call"] == "batch":
            out.append(("powerlaw", rows, 2 * 32 ** v, seed + 10 * i))
        else:
            out.append(("random" if i % 2 else "powerlaw", rows, 2 + 14 * v, seed + 10 * i))
    return out


def _requests(c):
    """(matrix, width) of each request to a server."""
    return [(i % c["matrices"], SERVE_WIDTHS[(i + i // c["matrices"]) % 3])
            for i in range(c["requests"])]


def prepare(case, seed):
    c, seed = case, 1000 * seed
    s = dict(case=c)
    if c["call"] == "batch":
        inst = []
        for kind, rows, degree, sd in _instances(c, seed):
            A, B = _matrix(kind, rows, degree, sd), _dense(rows, c["n"], sd + 1)
            d = dict(A=A, nv=c["n"], C=torch.empty(rows, c["n"], device="cuda"),
                     values=A.values.to(TORCH[c["val"]]), val_fmt=FORMATS[c["val"]],
                     b_fmt=FORMATS[c["b"]])
            if c["b"] == "e4m3":
                q, d["b_scales"] = _to_e4m3(B)
                d["B"] = q.view(torch.uint8)
            else:
                d["B"] = B.to(TORCH[c["b"]])
            inst.append(d)
        s.update(batch=D.Batch(inst), C=[d["C"] for d in inst])
        return s
    if c["call"] == "serve":
        s["server"] = D.Server(budget_bytes=1 << 29, b_fmt=FORMATS["bf16"])
        mats = _instances(c, seed)
        for m in mats:
            s["server"].add_matrix(_matrix(*m))
        s["requests"] = [(m, n, _dense(mats[m][1], n, mats[m][3] + n, "bf16"))
                         for m, n in _requests(c)]
        s["C"] = [torch.empty(mats[m][1], n, device="cuda") for m, n in _requests(c)]
        torch.cuda.synchronize()  # the server has a stream of its own
        return s
    A = _matrix(c["matrix"], c["rows"], c["degree"], seed)
    C, B = _operands(c, seed)
    s.update(A=A, B=B, C=C)
    if c["call"] == "mixed":
        s["values"] = A.values.to(TORCH[c["val"]])
        if not c["quantize"]:
            if c["b"] == "e4m3":
                q, s["scales"] = _to_e4m3(B)
                s["B"] = q.view(torch.uint8)
            else:
                s["B"], s["scales"] = B.to(TORCH[c["b"]]), None
    elif c["call"] == "plan":
        s["plan"] = D.Plan(A, c["n"])
    return s


def run(state):
    s, c = state, state["case"]
    if c["call"] == "spmm":
        D.spmm(ALGS[c["alg"]], int(c["layout"] == "col"), s["A"], s["B"], s["C"], beta=c["beta"],
               nv=c["n"])
    elif c["call"] == "compat":
        status = D.compat_spmm(ALGS[c["alg"]], int(c["layout"] == "col"), s["A"], s["B"], s["C"],
                               c["n"])
        if status:
            raise D.DaspmmError(3, f"cudaError {status}")
    elif c["call"] == "plan":
        s["plan"].spmm(s["B"], s["C"])
    elif c["call"] == "batch":
        s["batch"].run()
    elif c["call"] == "mixed":
        B, scales = s["B"], s.get("scales")
        if c["quantize"]:
            fmt, n = FORMATS[c["b"]], c["n"]
            scales = D.e4m3_scales(B, c["rows"], n) if c["b"] == "e4m3" else None
            B = D.quantize(B, fmt, scales, n if c["b"] == "e4m3" else 0)
        D.spmm_mixed(s["A"], s["values"], FORMATS[c["val"]], B, FORMATS[c["b"]], s["C"], c["n"],
                     b_scales=scales, beta=c["beta"])
        if c["quantize"]:
            return {"C": s["C"], "B": B.view(torch.uint8)}
    else:
        srv = s["server"]
        tickets = [srv.submit(*r) for r in s["requests"]]
        for t, C in zip(tickets, s["C"]):
            status, res = srv.wait(t)
            D.check(status or res.status, "serve")
            C.view(-1).copy_(srv.result_tensor(res, *C.shape))
        torch.cuda.current_stream().synchronize()  # the arena is given back
        for t in tickets:
            srv.release(t)
    return {"C": s["C"]}


# ------------------------------------------------------------------ what a pass cannot do without
def _bytes(kind, rows, degree, n, val, b, out=1, index_rows=False):
    nnz = rows * degree
    # columns that the matrix has at least one entry in
    used = rows * (degree / (1 + degree) if kind == "powerlaw" else 1 - math.exp(-degree))
    return (nnz * (4 + val) + 4 * (nnz if index_rows else rows + 1) + used * n * b
            + 4 * rows * n * out)


def work(case):
    c = case
    size = {"f32": 4, "bf16": 2, "f16": 2, "e4m3": 1}
    if c["call"] == "batch":
        inst = [(k, r, d, c["n"], size[c["val"]], size[c["b"]]) for k, r, d, _ in _instances(c, 0)]
    elif c["call"] == "serve":
        mats = _instances(c, 0)
        inst = [(*mats[m][:3], n, 4, 2) for m, n in _requests(c)]
        # each result is also read and written once where the caller takes it
        copies = sum(8 * mats[m][1] * n for m, n in _requests(c))
    else:
        m = (c["matrix"], c["rows"], c["degree"], c["n"])
        flops = 2 * c["rows"] * c["degree"] * c["n"]
        out = 2 if c.get("beta", 0.0) != 0.0 or c.get("alg", "").startswith("coo") else 1
        if c["call"] == "mixed":
            nbytes = _bytes(*m, size[c["val"]], size[c["b"]], out)
            if c["quantize"]:  # the float32 operand read, the codes written
                nbytes += c["rows"] * c["n"] * (4 + size[c["b"]])
        else:
            nbytes = _bytes(*m, 4, 4, out, c.get("alg", "").startswith("coo"))
        return {"bytes": nbytes, "flops": flops}
    return {"bytes": sum(_bytes(*i) for i in inst) + (copies if c["call"] == "serve" else 0),
            "flops": sum(2 * i[1] * i[2] * i[3] for i in inst)}


# ------------------------------------------------------------------ the same in 64 bits
def _product(csr, values, B):
    ptr, col, _ = csr
    rows = ptr.numel() - 1
    A = torch.sparse_csr_tensor(ptr.long(), col.long(), values.double(), (rows, rows))
    return A @ B.double()


def exact(case, seed):
    c, seed = case, 1000 * seed
    if c["call"] == "batch":
        out = []
        for kind, rows, degree, sd in _instances(c, seed):
            m, B = _csr(kind, rows, degree, sd), _dense(rows, c["n"], sd + 1)
            if c["b"] == "e4m3":
                q, scale = _to_e4m3(B)
                B = q.double() * scale.double()
            else:
                B = B.to(TORCH[c["b"]])
            out.append(_product(m, m[2].to(TORCH[c["val"]]), B))
        return {"C": out}
    if c["call"] == "serve":
        mats = _instances(c, seed)
        csr = [_csr(*m) for m in mats]
        return {"C": [_product(csr[m], csr[m][2], _dense(mats[m][1], n, mats[m][3] + n, "bf16"))
                      for m, n in _requests(c)]}
    m = _csr(c["matrix"], c["rows"], c["degree"], seed)
    C, B = _operands(c, seed)
    if c["call"] == "mixed":
        if c["b"] == "e4m3":
            q, scale = _to_e4m3(B)
            B = q.double() * scale.double()
        else:
            B = B.to(TORCH[c["b"]])
        values = m[2].to(TORCH[c["val"]])
    else:
        values = m[2]
    col = c.get("layout", "row") == "col"
    out = _product(m, values, B.t() if col else B)
    out = out.t().contiguous() if col else out
    beta = 1.0 if c["call"] == "compat" and c["alg"].startswith("coo") else c.get("beta", 0.0)
    if beta != 0.0:
        out += beta * C.double()
    return {"C": out, "B": None} if c["call"] == "mixed" and c["quantize"] else {"C": out}
