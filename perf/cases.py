"""The work that users of this framework have it do, as cases to be timed.

Sparse operands are the matrices of the five benchmark configurations (R-MAT graphs and rows of 16 uniformly drawn
columns) and ragged rectangular ones; dense operands are U(-1, 1).  The device cases are the calls a program makes
whose operands stay in GPU memory (``comet_b200.device``); the host cases are the calls COMET's generated code and
cometpy make, on numpy arrays (``comet_b200.api``), and are timed with the copies that belong to them.
"""
import math

import numpy as np
import torch

from comet_b200 import api, device

RMAT = (0.57, 0.19, 0.19, 0.05)          # quadrant probabilities of every graph here
INDEX = {"i64": np.int64, "i32": np.int32}
VALUE = {"f64": np.float64, "f32": np.float32}


def listed():
    return [
        # Configuration 1: a small solver-like matrix, multiplied again and again. Latency and launches count.
        {"name": "spmv_small", "op": "spmv", "matrix": "even", "rows": 16384, "cols": 16384, "per_row": 16},
        # One step of an iterative method (PageRank, power iteration) on a graph with hubs.
        {"name": "spmv_graph", "op": "spmv", "matrix": "rmat", "scale": 20, "edge_factor": 16},
        # Configuration 2: a graph times a block of 128 dense columns (features, block Krylov vectors).
        {"name": "spmm_graph_k128", "op": "spmm", "matrix": "rmat", "scale": 20, "edge_factor": 16, "k": 128},
        # Rectangular, rows of very different lengths, an odd number of narrow columns.
        {"name": "spmm_ragged_k33", "op": "spmm", "matrix": "ragged", "rows": 50021, "cols": 30011, "per_row": 12, "k": 33},
        # Configuration 3: sampled dense-dense product on a graph (attention scores, factorisation residuals).
        {"name": "sddmm_graph_k64", "op": "sddmm", "matrix": "rmat", "scale": 18, "edge_factor": 32, "k": 64},
        # A product of short rows, as in a multigrid set-up.
        {"name": "spgemm_even", "op": "spgemm", "matrix": "even", "rows": 16384, "cols": 16384, "per_row": 16, "semiring": "+,*"},
        # Configuration 4: a graph squared; nearly all of the traffic is the result.
        {"name": "spgemm_graph", "op": "spgemm", "matrix": "rmat", "scale": 18, "edge_factor": 16, "semiring": "+,*"},
        # Triangles per edge (truss decomposition): the masked product with its result stored.
        {"name": "spgemm_masked", "op": "spgemm_masked", "matrix": "symmetric", "scale": 15, "edge_factor": 16, "semiring": "+,pair"},
        # Configuration 5: triangle counting.
        {"name": "triangles_graph", "op": "triangles", "matrix": "lower", "scale": 22, "edge_factor": 16},
        # An edge list read from a file becomes a CSR matrix (the reader's sort; repeated entries stay).
        {"name": "host_coo_to_csr", "op": "host_coo_to_csr", "scale": 18, "entries": 4194301},
        # cometpy's A @ B on scipy's arrays (32-bit indices): upload, product, download.
        {"name": "host_spmm_k64", "op": "host_spmm", "matrix": "rmat", "scale": 17, "edge_factor": 16, "k": 64, "index": "i32", "value": "f64"},
        # The same for a vector and the matrix of configuration 1, as COMET's generated code calls it.
        {"name": "host_spmv_small", "op": "host_spmv", "matrix": "even", "rows": 16384, "cols": 16384, "per_row": 16, "index": "i64", "value": "f64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the same calls over the sizes, shapes and options between the smallest and the largest."""
    op = rng.choice(["spmv", "spmm", "sddmm", "spgemm", "spgemm_masked", "triangles", "host_coo_to_csr", "host_spmm",
                     "host_spmv"])
    c = {"op": op}
    if op == "host_coo_to_csr":
        return dict(c, scale=rng.randint(10, 20), entries=_log(rng, 1000, 4200000))
    if op == "spgemm_masked":
        return dict(c, matrix="symmetric", scale=rng.randint(9, 16), edge_factor=rng.randint(4, 16),
                    semiring=rng.choice(["+,pair", "+,*"]))
    if op == "triangles":
        return dict(c, matrix="lower", scale=rng.randint(9, 21), edge_factor=rng.randint(4, 16))
    c["matrix"] = rng.choice(["even", "ragged", "rmat", "rmat"])
    if c["matrix"] == "rmat":
        top = {"spgemm": 17, "host_spmm": 17, "host_spmv": 18}.get(op, 20)
        c.update(scale=rng.randint(10, top), edge_factor=rng.randint(4, 16))
        rows, entries = 1 << c["scale"], c["edge_factor"] << c["scale"]
    else:
        top = {"spgemm": 200000, "host_spmm": 200000, "host_spmv": 400000}.get(op, 1000000)
        rows = _log(rng, 1000, top)
        cols = rows if op == "spgemm" or rng.random() < 0.5 else _log(rng, 1000, top)
        c.update(rows=rows, cols=cols, per_row=_log(rng, 2, 32 if op == "spgemm" else 64))
        entries = rows * c["per_row"]
    if op == "spgemm":
        c["semiring"] = rng.choice(["+,*", "+,*", "+,*", "min,+"])
    if op in ("spmm", "sddmm", "host_spmm"):
        # no more products than the largest listed case of its kind
        top = {"spmm": 2e9, "sddmm": 5e8, "host_spmm": 1.3e8}[op] / max(entries, rows)
        c["k"] = max(1, min(_log(rng, 4, 256), int(top)))
        if rng.random() < 0.5:
            c["k"] += c["k"] % 2
    if op.startswith("host"):
        c.update(index=rng.choice(["i32", "i64"]), value=rng.choice(["f64", "f64", "f32"]))
    return c


# --- inputs ------------------------------------------------------------------------------------------------------

def _uniform(gen, shape, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _rmat_edges(gen, scale, entries):
    a, b, c, _ = RMAT
    rows = torch.zeros(entries, dtype=torch.int64, device="cuda")
    cols = torch.zeros(entries, dtype=torch.int64, device="cuda")
    for _level in range(scale):
        u = torch.rand(entries, generator=gen, device="cuda")
        rows.mul_(2).add_(u >= a + b)
        cols.mul_(2).add_(((u >= a) & (u < a + b)) | (u >= a + b + c))
    return rows, cols


def _permuted_bits(ids, order):
    out = torch.zeros_like(ids)
    for to, bit in enumerate(order):
        out |= ((ids >> bit) & 1) << to
    return out


def _pattern(case, gen, relabel):
    """Rows and columns of a matrix's entries (some of them more than once).  With ``relabel`` the pattern is the
    case's own and only its rows and columns are renumbered from ``gen``, so that every seed's product has as many
    entries.  The R-MAT levels are alike and the other matrices' rows too, so a renumbered one (levels in another order,
    rows and columns shuffled) is another draw from the same distribution."""
    kind = case["matrix"]
    draws = gen
    if relabel:
        draws = torch.Generator(device="cuda")
        draws.manual_seed(1)
    if kind in ("rmat", "symmetric", "lower"):
        r, c = _rmat_edges(draws, case["scale"], case["edge_factor"] << case["scale"])
        if relabel:
            order = torch.randperm(case["scale"], generator=gen, device="cuda").tolist()
            r, c = _permuted_bits(r, order), _permuted_bits(c, order)
        keep = r != c
        r, c = r[keep], c[keep]
        if kind == "symmetric":
            r, c = torch.cat([r, c]), torch.cat([c, r])
        elif kind == "lower":    # strict lower triangle of the symmetrised graph
            r, c = torch.maximum(r, c), torch.minimum(r, c)
        return r, c
    nrows, ncols, per = case["rows"], case["cols"], case["per_row"]
    if kind == "even":           # exactly per_row distinct columns in every row
        c = torch.randint(0, ncols - per + 1, (nrows, per), generator=draws, device="cuda")
        c = (torch.sort(c, 1)[0] + torch.arange(per, device="cuda")).reshape(-1)
        r = torch.arange(nrows, device="cuda").repeat_interleave(per)
    else:                        # rows of up to 2 per_row entries, empty ones among them
        lens = torch.randint(0, 2 * per + 1, (nrows,), generator=draws, device="cuda")
        r = torch.arange(nrows, device="cuda").repeat_interleave(lens)
        c = torch.randint(0, ncols, (r.numel(),), generator=draws, device="cuda")
    if relabel:
        rp = torch.randperm(nrows, generator=gen, device="cuda")
        cp = rp if nrows == ncols else torch.randperm(ncols, generator=gen, device="cuda")
        r, c = rp[r], cp[c]
    return r, c


def _matrix(case, gen):
    # triangle counts do not depend on the numbering, so there the seed draws the graph itself
    r, c = _pattern(case, gen, relabel=case["op"] != "triangles")
    nrows = case["rows"] if "rows" in case else 1 << case["scale"]
    ncols = case["cols"] if "cols" in case else nrows
    keys = torch.sort(r * ncols + c)[0]
    del r, c
    if keys.numel() > 1:
        keys = keys[torch.cat([keys.new_ones(1, dtype=torch.bool), keys[1:] != keys[:-1]])]
    r = torch.div(keys, ncols, rounding_mode="floor")
    crd = keys - r * ncols
    pos = torch.zeros(nrows + 1, dtype=torch.int64, device="cuda")
    pos[1:] = torch.cumsum(torch.bincount(r, minlength=nrows), 0)
    if case["matrix"] == "lower" or case.get("semiring") == "+,pair":
        val = torch.ones(crd.numel(), dtype=torch.float64, device="cuda")
    elif case["matrix"] in ("rmat", "symmetric"):
        val = _uniform(gen, crd.numel(), 0.5, 1.5)
    else:
        val = _uniform(gen, crd.numel())
    return device.DeviceCSR(nrows, ncols, pos, crd, val)


def _to_host(A, case):
    it, vt = INDEX[case["index"]], VALUE[case["value"]]
    host = lambda t, dt: t.cpu().numpy().astype(dt)
    return api.SparseTensor("CSR", A.nrows, A.ncols, np.array([A.nrows], dtype=it), np.array([-1], dtype=it),
                            host(A.pos, it), host(A.crd, it), host(A.val, vt))


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op = case["op"]
    if op == "host_coo_to_csr":
        n = 1 << case["scale"]
        r, c = _rmat_edges(gen, case["scale"], case["entries"])
        v = _uniform(gen, case["entries"])
        return {"op": op, "rows": r.cpu().numpy(), "cols": c.cpu().numpy(), "vals": v.cpu().numpy(), "shape": (n, n)}
    A = _matrix(case, gen)
    s = {"op": op, "A": A, "semiring": case.get("semiring")}
    if op in ("spmv", "host_spmv"):
        s["x"] = _uniform(gen, A.ncols)
    elif op in ("spmm", "host_spmm"):
        s["B"] = _uniform(gen, (A.ncols, case["k"]))
    elif op == "sddmm":
        s["X"], s["Y"] = _uniform(gen, (A.nrows, case["k"])), _uniform(gen, (A.ncols, case["k"]))
    if op.startswith("host"):
        s["A"] = _to_host(A, case)
        for name in ("x", "B"):
            if name in s:
                s[name] = s[name].cpu().numpy().astype(VALUE[case["value"]])
    return s


# --- the calls ---------------------------------------------------------------------------------------------------

_SEMIRING = {"+,*": api.PLUS_TIMES, "+,pair": api.PLUS_PAIR, "min,+": api.MIN_PLUS}


def run(s):
    op, A = s["op"], s.get("A")
    if op == "spmv":
        return device.spmv(A, s["x"])
    if op == "spmm":
        return device.spmm(A, s["B"])
    if op == "sddmm":
        return device.sddmm(A, s["X"], s["Y"])
    if op == "spgemm":
        C = device.spgemm(A, A, semiring=_SEMIRING[s["semiring"]])
        return C.pos, C.crd, C.val
    if op == "spgemm_masked":
        C = device.spgemm(A, A, A, semiring=_SEMIRING[s["semiring"]])
        return C.pos, C.crd, C.val
    if op == "triangles":
        return device.masked_pair_count(A, A, A)
    if op == "host_coo_to_csr":
        C = api.from_coordinates(s["rows"], s["cols"], s["vals"], s["shape"])
        return C.a2pos, C.a2crd, C.val
    if op == "host_spmm":
        return api.spmm(A, s["B"])
    return api.spmv(A, s["x"])


# --- what a call cannot do without -------------------------------------------------------------------------------

def _classes(scale, edges):
    """R-MAT cells by (zero bits of the row, zero bits of the column): yields row bits, column bits, number of such
    cells and the expected number of distinct entries in one of them.  i levels draw quadrant a, j draw b, l draw c."""
    a, b, c, d = RMAT
    f = math.factorial
    for i in range(scale + 1):
        for j in range(scale + 1 - i):
            for l in range(scale + 1 - i - j):
                m = scale - i - j - l
                cells = f(scale) // (f(i) * f(j) * f(l) * f(m))
                yield i + j, i + l, cells, -math.expm1(-edges * a ** i * b ** j * c ** l * d ** m)


def _size(case):
    """Rows, columns, expected stored entries and expected products of A * A."""
    kind = case["matrix"]
    if kind in ("even", "ragged"):
        n = case["rows"] * case["per_row"]
        return case["rows"], case["cols"], n, n * case["per_row"]
    scale = case["scale"]
    edges = (case["edge_factor"] << scale) * (1 if kind == "rmat" else 2)     # b = c: both directions are as likely
    rows = [0.0] * (scale + 1)     # stored entries in the rows with z zero bits
    cols = [0.0] * (scale + 1)
    for zr, zc, cells, q in _classes(scale, edges):
        rows[zr] += cells * q
        cols[zc] += cells * q
    products = sum(r * c / math.comb(scale, z) for z, (r, c) in enumerate(zip(rows, cols)))
    return 1 << scale, 1 << scale, sum(rows) * (0.5 if kind == "lower" else 1), products


def work(case):
    op = case["op"]
    if op == "host_coo_to_csr":
        return {"bytes": 48 * case["entries"] + (8 << case["scale"]), "flops": 0}
    nrows, ncols, nnz, products = _size(case)
    iw = 4 if case.get("index") == "i32" else 8
    vw = 4 if case.get("value") == "f32" else 8
    sparse = iw * (nrows + 1) + (iw + vw) * nnz
    if op in ("spmv", "host_spmv"):
        return {"bytes": sparse + vw * (nrows + ncols), "flops": 2 * nnz}
    if op in ("spmm", "host_spmm"):
        return {"bytes": sparse + vw * (nrows + ncols) * case["k"], "flops": 2 * nnz * case["k"]}
    if op == "sddmm":
        return {"bytes": sparse + 8 * nnz + 8 * (nrows + ncols) * case["k"], "flops": nnz * (2 * case["k"] + 1)}
    if op == "triangles":
        return {"bytes": 8 * (nrows + 1) + 8 * nnz, "flops": 2 * nnz}
    if op == "spgemm_masked":
        return {"bytes": 2 * sparse, "flops": 2 * nnz}
    if case["matrix"] == "rmat":   # the result, as if its entries met at random in each class of cells
        a, b, c, d = RMAT
        p2 = (a * a + b * c, a * b + b * d, c * a + d * c, c * b + d * d)
        f, scale = math.factorial, case["scale"]
        edges = float(case["edge_factor"] << scale)
        out = 0.0
        for i in range(scale + 1):
            for j in range(scale + 1 - i):
                for l in range(scale + 1 - i - j):
                    m = scale - i - j - l
                    cells = f(scale) // (f(i) * f(j) * f(l) * f(m))
                    out -= cells * math.expm1(-edges * edges * p2[0] ** i * p2[1] ** j * p2[2] ** l * p2[3] ** m)
    else:
        out = nrows * ncols * -math.expm1(-products / (nrows * ncols))
    return {"bytes": sparse + 8 * (nrows + 1) + 16 * min(out, products), "flops": 2 * products}


def tolerance(case):
    """Structure, counts and moved values are exact; sums may be taken in another order."""
    if case["op"] in ("triangles", "host_coo_to_csr") or case.get("semiring") in ("+,pair", "min,+"):
        return "exact"
    if case.get("value") == "f32":
        return {"rel": 1e-6}
    return {"rel": 1e-12, "max": 1e-10}
