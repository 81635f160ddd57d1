"""Performance cases of casgemm: the work its users have it do, through its public Python entry points.

Each case is a dict of plain values.  `op` names the entry point:

  product    Context.spgemm_device: C = A * B on matrices resident on the device (C = A * A^T for the graphs)
  host       Context.spgemm: host CSR in, host CSR out
  transpose  Context.transpose_device: B = A^T, the second input when a program has A alone
  batch      Context.batch_run: many independent products, outputs kept as digests

and `family` the matrices:

  er      uniform random graph, `rows` vertices, `ef` undirected edges a vertex (R-MAT with a = b = c = d)
  g500    Graph500 R-MAT graph (a, b, c = 0.57, 0.19, 0.19), the same
  zipf    bipartite join matrix, row degrees Zipf(1.2) up to `amax`, column popularity Zipf(1.4) shifted by 1000
  ragged  A (rows x mid) times an independent B (mid x cols), row lengths exponential with means `ra` and `rb`

The structure of a matrix belongs to its case, so that C has as many entries for every seed; the seed shifts the
vertices (or the rows, the inner and the outer columns) cyclically, which keeps the neighbourhoods that the kernels
meet, and draws the values.

Values are `ones` (what the MatrixMarket loader gives every entry), `int` (int32 in 1..8, summed in int64) or
`normal` (fp64 reals).  Graph inputs are made on the device, since a program that calls these entry points holds its
matrices there.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "contention-aware-spgemm_b200"))
import casgemm  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest calls: a test-sized graph, where launches, waits and allocations are all there is
        {"name": "g500_256_hash", "op": "product", "family": "g500", "rows": 256, "ef": 4, "accum": "hash",
         "values": "ones"},
        # one job of the uneven batch on its own, int32 in and int64 out
        {"name": "g500_4k_int", "op": "product", "family": "g500", "rows": 4096, "ef": 16, "accum": "hsersc",
         "values": "int"},
        # an ordinary skewed graph of a vertex count that is no power of two, reals for values
        {"name": "g500_27k_real", "op": "product", "family": "g500", "rows": 27001, "ef": 8, "accum": "hybacc",
         "values": "normal"},
        # the Graph500 configuration: scale 17, edge factor 8, hybrid accumulator
        {"name": "g500_131k", "op": "product", "family": "g500", "rows": 131072, "ef": 8, "accum": "hybacc",
         "values": "ones"},
        # sparse uniform graph: rows of 16 products, the warp-sized kernels
        {"name": "er_500k_tiny", "op": "product", "family": "er", "rows": 500009, "ef": 2, "accum": "hash",
         "values": "ones"},
        # uniform graph with rows of 256 products: the small ESC rows and their symbolic pass
        {"name": "er_131k_small", "op": "product", "family": "er", "rows": 131072, "ef": 8, "accum": "hsersc",
         "values": "ones"},
        # the headline's shape (edge factor 32, rows of about 4096 products) at the largest size whose C fits the
        # card three times over
        {"name": "er_524k", "op": "product", "family": "er", "rows": 524288, "ef": 32, "accum": "hybacc",
         "values": "ones"},
        # the join-aggregate configuration's shape: heavy rows over more than one column slice
        {"name": "zipf_600k", "op": "product", "family": "zipf", "rows": 600000, "cols": 1400000, "nnz": 6000000,
         "amax": 25000, "accum": "hybacc", "values": "ones"},
        # general A * B with ragged rows, odd sizes and real values
        {"name": "ragged_70k", "op": "product", "family": "ragged", "rows": 70001, "mid": 90007, "cols": 250013,
         "ra": 11, "rb": 37, "accum": "hybacc", "values": "normal"},
        # B = A^T on the device before the product of a program that has A alone
        {"name": "transpose_g500_262k", "op": "transpose", "family": "g500", "rows": 262144, "ef": 16,
         "values": "ones"},
        # many small jobs in one call: the batch's scales 10 to 13
        {"name": "batch_32", "op": "batch", "jobs": 32, "lo": 1024, "hi": 8192, "mode": "waves", "values": "int"},
        # a program whose matrices are in host memory, as the drivers' are
        {"name": "host_er_16k", "op": "host", "family": "er", "rows": 16384, "ef": 8, "accum": "hybacc",
         "values": "ones"},
    ]


# ----------------------------------------------------------------- drawn cases
MOST_PRODUCTS = 1.2e9  # below the largest listed case's


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _products(family, rows, ef):
    """About how many products A * A^T has (an upper bound for the skewed graphs)."""
    if family == "er":
        return 4.0 * ef * ef * rows
    return 4.0 * ef * ef * rows * rows * 0.6352 ** math.log2(rows)


def _draw_graph(rng, most):
    while True:
        family = rng.choice(["er", "g500"])
        rows, ef = _log_uniform(rng, 200, 600000), _log_uniform(rng, 1, 40)
        if rows >= 16 * ef and _products(family, rows, ef) <= most:
            return {"family": family, "rows": rows, "ef": ef}


def draw(rng):
    op = rng.choice(["product"] * 11 + ["transpose", "batch", "host"])
    accum = rng.choice(["hybacc", "hybacc", "hsersc", "hash"])
    values = rng.choice(["ones", "ones", "normal", "int"])
    if op == "batch":
        lo = _log_uniform(rng, 500, 2000)
        return {"op": op, "jobs": rng.randint(8, 48), "lo": lo, "hi": lo * rng.randint(2, 6), "mode": "waves",
                "values": "int"}
    if op == "transpose":
        return dict({"op": op, "values": values}, **_draw_graph(rng, 1e12))
    if op == "host":
        return dict({"op": op, "accum": accum, "values": values}, **_draw_graph(rng, 5e6))
    kind = rng.choice(["graph"] * 7 + ["ragged"] * 3 + ["zipf"])
    if kind == "zipf":
        rows = _log_uniform(rng, 30000, 500000)
        return {"op": op, "family": "zipf", "rows": rows, "cols": int(rows * rng.uniform(1.5, 3.0)),
                "nnz": int(rows * rng.uniform(4.0, 9.0)), "amax": max(500, rows // rng.randint(20, 60)), "accum": accum,
                "values": rng.choice(["ones", "int"])}
    if kind == "ragged":
        while True:
            rows, mid, cols = (_log_uniform(rng, 300, 300000) for _ in range(3))
            ra, rb = _log_uniform(rng, 2, 100), _log_uniform(rng, 2, 100)
            if mid >= 8 * ra and cols >= 8 * rb and rows * ra * rb <= 2e8:
                return {"op": op, "family": "ragged", "rows": rows, "mid": mid, "cols": cols, "ra": ra, "rb": rb,
                        "accum": accum, "values": values}
    return dict({"op": op, "accum": accum, "values": values}, **_draw_graph(rng, MOST_PRODUCTS))


# -------------------------------------------------------------------- matrices
class Matrix:
    """A CSR in torch tensors on the device, columns ascending and distinct in every row."""

    def __init__(self, nrow, ncol, rp, cols, vals):
        self.nrow, self.ncol, self.rp, self.cols, self.vals = nrow, ncol, rp, cols, vals

    @property
    def nnz(self):
        return self.cols.numel()

    def rows(self):
        return torch.repeat_interleave(torch.arange(self.nrow, device=DEV), self.rp[1:] - self.rp[:-1])

    def device_csr(self):
        vt = casgemm.VAL_I32 if self.vals.dtype == torch.int32 else casgemm.VAL_F64
        return casgemm.DeviceCsr(self.nrow, self.ncol, self.nnz, self.rp.data_ptr(), self.cols.data_ptr(),
                                 self.vals.data_ptr(), vt, keep=self)

    def host_csr(self):
        return casgemm.Csr(self.nrow, self.ncol, self.rp.cpu().numpy(), self.cols.cpu().numpy(),
                           self.vals.cpu().numpy())


def _values(nnz, values, gen):
    if values == "int":
        return torch.randint(1, 9, (nnz,), dtype=torch.int32, device=DEV, generator=gen)
    if values == "normal":
        return torch.randn(nnz, dtype=torch.float64, device=DEV, generator=gen)
    return torch.ones(nnz, dtype=torch.float64, device=DEV)


def _from_keys(nrow, ncol, key, values, gen, rshift, cshift):
    """CSR of the distinct keys row * ncol + col, rows and columns shifted cyclically."""
    row = key // ncol
    key = torch.sort((row + rshift) % nrow * ncol + (key - row * ncol + cshift) % ncol).values
    row = key // ncol
    rp = torch.zeros(nrow + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.bincount(row, minlength=nrow).cumsum(0)
    return Matrix(nrow, ncol, rp, (key - row * ncol).to(torch.int32), _values(key.numel(), values, gen))


def _transpose(M):
    order = torch.sort(M.cols, stable=True).indices
    rp = torch.zeros(M.ncol + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.bincount(M.cols, minlength=M.ncol).cumsum(0)
    return Matrix(M.ncol, M.nrow, rp, M.rows()[order].to(torch.int32), M.vals[order])


def _graph(family, n, ef, values, gen, made, shift):
    """Symmetric graph of n vertices and n * ef distinct undirected edges, no loops."""
    want, have = n * ef, torch.empty(0, dtype=torch.int64, device=DEV)
    bits = max(1, (n - 1).bit_length())
    for _ in range(40):
        e = int((want - have.numel()) * 1.1) + 64
        if family == "er":
            r = torch.randint(0, n, (e,), device=DEV, generator=made)
            c = torch.randint(0, n, (e,), device=DEV, generator=made)
        else:
            r = torch.zeros(e, dtype=torch.int64, device=DEV)
            c = torch.zeros(e, dtype=torch.int64, device=DEV)
            for _ in range(bits):
                u = torch.rand(e, device=DEV, generator=made)
                r = r * 2 + (u >= 0.76)
                c = c * 2 + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
        ok = (r != c) & (r < n) & (c < n)
        r, c = r[ok], c[ok]
        have = torch.unique(torch.cat([have, torch.minimum(r, c) * n + torch.maximum(r, c)]))
        if have.numel() >= want:
            break
    if have.numel() > want:
        have = have[torch.randperm(have.numel(), device=DEV, generator=made)[:want]]
    r, c = have // n, have % n
    return _from_keys(n, n, torch.cat([r * n + c, c * n + r]), values, gen, shift, shift)


def _zipf(nrow, ncol, nnz, amax, values, gen, made, rshift, cshift):
    """Row degrees amax * ((1 + q) / (r + q))^1.2 with q such that they sum to nnz, rows shuffled; columns drawn with
    probability falling as (k + 1000)^-1.4."""
    r = torch.arange(1, nrow + 1, dtype=torch.float64, device=DEV)

    def degrees(q):
        return (amax * ((1.0 + q) / (r + q)) ** 1.2).round().clamp(min=1)

    lo, hi = 0.0, 1.0
    while float(degrees(hi).sum()) < nnz and hi < 1e12:
        hi *= 2
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if float(degrees(mid).sum()) < nnz else (lo, mid)
    deg = degrees(hi).to(torch.int64)[torch.randperm(nrow, device=DEV, generator=made)]
    row = torch.repeat_interleave(torch.arange(nrow, device=DEV), deg)
    cdf = (torch.arange(1, ncol + 1, dtype=torch.float64, device=DEV) + 1000.0).pow(-1.4).cumsum(0)
    u = torch.rand(row.numel(), dtype=torch.float64, device=DEV, generator=made) * cdf[-1]
    col = torch.searchsorted(cdf, u).clamp(max=ncol - 1)
    return _from_keys(nrow, ncol, torch.unique(row * ncol + col), values, gen, rshift, cshift)


def _ragged(nrow, ncol, mean, values, gen, made, rshift, cshift):
    u = torch.rand(nrow, dtype=torch.float64, device=DEV, generator=made)
    deg = (-mean * torch.log1p(-u)).round().clamp(max=ncol // 2).to(torch.int64)
    row = torch.repeat_interleave(torch.arange(nrow, device=DEV), deg)
    col = torch.randint(0, ncol, (row.numel(),), device=DEV, generator=made)
    return _from_keys(nrow, ncol, torch.unique(row * ncol + col), values, gen, rshift, cshift)


def _matrices(case, seed):
    """(A, B) of a case; B is A itself for a symmetric graph with equal values, as a program would pass it."""
    gen, made = torch.Generator(device=DEV), torch.Generator(device=DEV)
    gen.manual_seed(seed * 1000003 + 17)
    made.manual_seed(case.get("graph", 0) + 29)
    rnd = np.random.default_rng(seed)
    family, values = case["family"], case["values"]
    s0, s1, s2 = (int(rnd.integers(1 << 40)) for _ in range(3))
    if family == "ragged":
        return (_ragged(case["rows"], case["mid"], case["ra"], values, gen, made, s0, s1),
                _ragged(case["mid"], case["cols"], case["rb"], values, gen, made, s1, s2))
    if family == "zipf":
        A = _zipf(case["rows"], case["cols"], case["nnz"], case["amax"], values, gen, made, s0, s1)
        return A, _transpose(A)
    A = _graph(family, case["rows"], case["ef"], values, gen, made, s0)
    return (A, A) if values == "ones" else (A, _transpose(A))


def _batch_jobs(case, seed):
    """[(A, B)] of the batch: sizes log-uniform over [lo, hi], edge factors 2 to 32, as in the uneven batch."""
    rnd = np.random.default_rng(5)
    jobs = []
    for j in range(case["jobs"]):
        n = int(round(math.exp(rnd.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        ef = int(rnd.choice([2, 4, 8, 16, 32]))
        one = {"family": "g500", "rows": n, "ef": ef, "values": case["values"], "graph": j}
        jobs.append(_matrices(one, seed * 4096 + j))
    return jobs


# ------------------------------------------------------------- prepare and run
_CTX = None


def _context():
    """The one context a program keeps."""
    global _CTX
    if _CTX is None:
        _CTX = casgemm.Context(0)
    return _CTX


class State:
    """What a program has in hand: its matrices, its context, and the C of its last call, which it gives back."""

    def __init__(self, case):
        self.case, self.ctx, self.C = case, _context(), None

    def release(self):
        if self.C is not None:
            self.ctx.free(self.C)
            self.C = None

    def __del__(self):
        try:
            self.release()
        except Exception:
            pass


def prepare(case, seed):
    s = State(case)
    if case["op"] == "batch":
        s.jobs = [(A.device_csr(), B.device_csr()) for A, B in _batch_jobs(case, seed)]
    else:
        A, B = _matrices(case, seed)
        if case["op"] == "host":
            s.A = A.host_csr()
            s.B = s.A if B is A else B.host_csr()
        else:
            s.A = A.device_csr()
            s.B = s.A if B is A else B.device_csr()
    torch.cuda.synchronize()  # the context works on a stream of its own
    return s


def run(s):
    op = s.case["op"]
    if op == "batch":
        jobs, _ = s.ctx.batch_run(s.jobs, accum="hybacc", mode=s.case["mode"], row_digests=True)
        return {"flop": np.array([j["flop"] for j in jobs], np.int64),
                "nnz_c": np.array([j["nnz_c"] for j in jobs], np.int64),
                "digest": np.array([j["digest"] for j in jobs], np.uint64),
                "row_digests": [j["row_digests"] for j in jobs]}
    if op == "host":
        C = s.ctx.spgemm(s.A, s.B, s.case["accum"]).csr
        return [C.row_ptrs, C.cols, C.vals]
    s.release()  # the C of the call before, as a program that is done with it does
    if op == "transpose":
        s.C = s.ctx.transpose_device(s.A)
    else:
        s.C, _ = s.ctx.spgemm_device(s.A, s.B, s.case["accum"])
    out = list(casgemm.device_tensors(s.C))
    for t in out:
        t.state = s  # the views are valid while the program keeps C
    return out


# --------------------------------------------------------------- work and exact
def _csr_bytes(nrow, nnz, vbytes):
    return 8.0 * (nrow + 1) + (4.0 + vbytes) * nnz


def _product_count(A, B):
    return int((B.rp[1:] - B.rp[:-1])[A.cols.long()].sum())


def work(case):
    """Each input once and each output once (a batch's outputs are its digests); two operations a product."""
    if case["op"] == "batch":
        by = fl = 0.0
        for A, B in _batch_jobs(case, 0):
            by += 2 * _csr_bytes(A.nrow, A.nnz, 4) + 8.0 * A.nrow
            fl += 2.0 * _product_count(A, B)
        return {"bytes": by, "flops": fl}
    A, B = _matrices(case, 0)
    v = A.vals.element_size()
    by = _csr_bytes(A.nrow, A.nnz, v)
    if case["op"] == "transpose":
        return {"bytes": by + _csr_bytes(A.ncol, A.nnz, v), "flops": 0.0}
    if B is not A:
        by += _csr_bytes(B.nrow, B.nnz, v)
    fl = 2.0 * _product_count(A, B)
    del A, B
    nnz_c = int(run(prepare(case, 0))[1].shape[0])
    return {"bytes": by + _csr_bytes(case["rows"], nnz_c, 8), "flops": fl}


EXACT_PRODUCTS = 1.5e8  # products that plain torch and numpy expand, sort and sum in some seconds


def _exact_product(A, B):
    """(row pointers, columns, values) of A * B: every product expanded, sorted by (row, column) and summed, whole
    numbers in int64 and reals in extended precision, rounded once."""
    rlen = (B.rp[1:] - B.rp[:-1])[A.cols.long()]
    n = int(rlen.sum())
    entry = torch.repeat_interleave(torch.arange(A.nnz, device=DEV), rlen)
    start = torch.cumsum(rlen, 0) - rlen
    at = B.rp[:-1][A.cols.long()][entry] + torch.arange(n, device=DEV) - start[entry]
    key = A.rows()[entry] * B.ncol + B.cols.long()[at]
    key, order = torch.sort(key, stable=True)
    entry, at = entry[order], at[order]
    uniq, counts = torch.unique_consecutive(key, return_counts=True)
    row = uniq // B.ncol
    rp = torch.zeros(A.nrow + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.bincount(row, minlength=A.nrow).cumsum(0)
    cols = (uniq - row * B.ncol).to(torch.int32)
    a, b = A.vals[entry], B.vals[at]
    first = (torch.cumsum(counts, 0) - counts).cpu().numpy()
    if a.dtype == torch.int32:
        p, kind = (a.long() * b.long()).cpu().numpy(), np.int64
    else:
        p, kind = a.cpu().numpy().astype(np.longdouble) * b.cpu().numpy(), np.float64
    vals = np.add.reduceat(p, first).astype(kind) if n else np.zeros(0, kind)
    return rp, cols, torch.from_numpy(vals)


def exact(case, seed):
    if case["op"] == "batch":
        jobs = _batch_jobs(case, seed)
        nnz = [int(_exact_product(A, B)[1].numel()) for A, B in jobs]
        return {"flop": np.array([_product_count(A, B) for A, B in jobs], np.int64), "nnz_c": np.array(nnz, np.int64),
                "digest": None, "row_digests": None}  # hashes of the rows: no numbers that have an error
    A, B = _matrices(case, seed)
    if case["op"] == "transpose":
        T = _transpose(A)
        return [T.rp, T.cols, T.vals]
    if _product_count(A, B) > EXACT_PRODUCTS:
        return None
    return list(_exact_product(A, B))
