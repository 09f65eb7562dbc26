"""The work that a program built on this package has it do, as cases that can be timed.

Every case goes through the package's public Python entry points on device data.
A case's "op" is one of

  multiply   y = A x or y += A x in one of the six formats
  vectors    the vector steps beside a multiply: dot, waxpby and reduce
  batch      many small CSR products in one persistent launch
  cg         conjugate gradients, a fixed number of iterations
  assemble   CSR from COO triplets in arbitrary order
  sort       COO triplets brought into (row, column) order
  convert    a row-sorted COO matrix to another format
  switch     a DynamicMatrix in CSR changes in place to the format that the selector picks

Matrices have the structures of the benchmark workloads: "stencil" is a 5-, 9-, 7- or
27-point stencil on an ni x nj (x nk) grid with 1e-3 jitter on the coefficients, optionally
with `offband` random entries per nonzero elsewhere; "power_law" has lognormal(2.0, 1.2) row
lengths clipped to [1, 4096] and uniform columns.  x is uniform in [-1, 1].
"""
import math

import torch

from morpheus_gb300 import batched, solvers
from morpheus_gb300.algorithms import dot, multiply, reduce, waxpby
from morpheus_gb300.containers import (COO_FORMAT, CSR_FORMAT, DIA_FORMAT, ELL_FORMAT, HDC_FORMAT, HYB_FORMAT,
                                       CooMatrix, CsrMatrix, DynamicMatrix)
from morpheus_gb300.convert import convert, from_coo, sort_by_row_and_column, to_coo

DEVICE = "cuda"
FORMATS = {"coo": COO_FORMAT, "csr": CSR_FORMAT, "dia": DIA_FORMAT, "ell": ELL_FORMAT, "hyb": HYB_FORMAT,
           "hdc": HDC_FORMAT}
DTYPES = {"f64": torch.float64, "f32": torch.float32}
MU, SIGMA, MAX_ROW = 2.0, 1.2, 4096
MEAN_ROW = math.exp(MU + SIGMA * SIGMA / 2)  # mean length of a power-law row
P90_ROW = 34                                 # nine rows in ten are no longer: the ELL width that HYB is given
LAM_LO, LAM_HI = 3.0, 40.0                   # mean row lengths of a batch's matrices


def listed():
    return [
        # One multiply of a matrix that a unit test or a coarse multigrid level has: latency.
        {"name": "multiply_csr_laplacian_32", "op": "multiply", "format": "csr", "structure": "stencil", "points": 5,
         "ni": 32, "nj": 32, "nk": 1, "offband": 0.0, "dtype": "f64", "init": True},
        # The vector steps of a hand-written solver on the 256 x 256 grid: three short calls, two of them
        # with a result that the host reads.
        {"name": "vectors_65536", "op": "vectors", "n": 65536, "dtype": "f64", "alpha": 1.0, "beta": -0.37},
        # A graph or circuit matrix in the default format, rows of very unequal length.
        {"name": "multiply_csr_power_law", "op": "multiply", "format": "csr", "structure": "power_law",
         "nrows": 2000000, "dtype": "f64", "init": True},
        # The same kind of matrix as triplets, in single precision.
        {"name": "multiply_coo_power_law_f32", "op": "multiply", "format": "coo", "structure": "power_law",
         "nrows": 2000000, "dtype": "f32", "init": True},
        # The same kind split into ELL and COO parts, added to y (a residual), an odd number of rows.
        {"name": "multiply_hyb_power_law_add", "op": "multiply", "format": "hyb", "structure": "power_law",
         "nrows": 1234567, "dtype": "f64", "init": False},
        # The 27-point stencil on 160^3, the benchmark's headline, in the format that the selector picks.
        {"name": "multiply_dia_stencil_160", "op": "multiply", "format": "dia", "structure": "stencil", "points": 27,
         "ni": 160, "nj": 160, "nk": 160, "offband": 0.0, "dtype": "f64", "init": True},
        # The same stencil where the program stays with CSR, in single precision.
        {"name": "multiply_csr_stencil_160_f32", "op": "multiply", "format": "csr", "structure": "stencil",
         "points": 27, "ni": 160, "nj": 160, "nk": 160, "offband": 0.0, "dtype": "f32", "init": True},
        # A stencil with a percent of couplings off its diagonals on a grid of odd sides.
        {"name": "multiply_hdc_offband_ragged", "op": "multiply", "format": "hdc", "structure": "stencil",
         "points": 27, "ni": 101, "nj": 97, "nk": 103, "offband": 0.01, "dtype": "f64", "init": True},
        # Many small independent systems, tuned once and multiplied in one launch.
        {"name": "batch_4096", "op": "batch", "count": 4096, "nmin": 64, "nmax": 8192, "dtype": "f64"},
        # A device-resident solve on the 2-D Laplacian.
        {"name": "cg_laplacian_2048", "op": "cg", "ni": 2048, "nj": 2048, "iters": 64, "dtype": "f64"},
        # A matrix put together from element or edge contributions in the order that they were found.
        {"name": "assemble_power_law", "op": "assemble", "structure": "power_law", "nrows": 1000000, "dtype": "f64"},
        # Format selection and the conversion that it asks for, on the headline matrix.
        {"name": "switch_stencil_160", "op": "switch", "structure": "stencil", "points": 27, "ni": 160, "nj": 160,
         "nk": 160, "offband": 0.0, "dtype": "f64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_stencil(rng, most):
    points = rng.choice([5, 9, 7, 27])
    n = _log_int(rng, 500, most // points)
    if points in (5, 9):
        ni = max(8, int(round(math.sqrt(n) * rng.uniform(0.7, 1.4))))
        nj, nk = max(8, n // ni), 1
    else:
        ni = max(6, int(round(n ** (1 / 3) * rng.uniform(0.8, 1.2))))
        nj = max(6, int(round(math.sqrt(n / ni) * rng.uniform(0.9, 1.1))))
        nk = max(6, n // (ni * nj))
    return {"structure": "stencil", "points": points, "ni": ni, "nj": nj, "nk": nk, "offband": 0.0}


def draw(rng):
    dtype = rng.choice(["f64", "f64", "f32"])
    op = rng.choice(["multiply"] * 6 + ["vectors", "batch", "cg", "assemble", "sort", "convert", "convert", "switch"])
    if op == "vectors":
        alpha, beta = rng.choice([(1.0, rng.uniform(-1, 1)), (rng.uniform(-1, 1), 1.0),
                                  (rng.uniform(-1, 1), rng.uniform(-1, 1))])
        return {"op": op, "n": _log_int(rng, 1000, 60_000_000), "dtype": dtype, "alpha": alpha, "beta": beta}
    if op == "batch":
        nmin = _log_int(rng, 32, 512)
        return {"op": op, "count": _log_int(rng, 64, 4096), "nmin": nmin,
                "nmax": min(8192, nmin * _log_int(rng, 4, 64)), "dtype": dtype}
    if op == "cg":
        n = _log_int(rng, 4000, 4_000_000)  # far from convergence after these iterations
        ni = max(8, int(round(math.sqrt(n) * rng.uniform(0.7, 1.4))))
        return {"op": op, "ni": ni, "nj": max(8, n // ni), "iters": rng.randint(8, 24), "dtype": "f64"}
    if op in ("assemble", "sort"):
        case = _draw_stencil(rng, 20_000_000) if rng.random() < 0.5 else \
            {"structure": "power_law", "nrows": _log_int(rng, 1000, 1_000_000)}
        return {"op": op, **case, "dtype": dtype}
    power_law = {"structure": "power_law", "nrows": _log_int(rng, 1000, 2_000_000)}
    if op == "switch":
        case = _draw_stencil(rng, 100_000_000) if rng.random() < 0.7 else power_law
        return {"op": op, **case, "dtype": dtype}
    if rng.random() < 0.5:
        case, formats = power_law, ["csr", "coo", "hyb"]
    else:
        case, formats = _draw_stencil(rng, 100_000_000), ["csr", "coo", "dia", "ell", "hdc"]
        case["offband"] = rng.choice([0.0, 0.0, 0.01, 0.03])
        if case["offband"]:
            formats = ["csr", "coo", "hdc", "hdc"]
    if op == "convert":
        return {"op": op, "format": rng.choice([f for f in formats if f != "coo"]), **case, "dtype": dtype}
    return {"op": op, "format": rng.choice(formats), **case, "dtype": dtype, "init": rng.random() < 0.7}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _normal(g, n, dtype):
    v = torch.randn(n, generator=g, device=DEVICE, dtype=dtype)
    v[v == 0] = 1.0
    return v


def _uniform(g, n, dtype, lo=-1.0, hi=1.0):
    return torch.rand(n, generator=g, device=DEVICE, dtype=dtype) * (hi - lo) + lo


def _offsets(points):
    one = (-1, 0, 1)
    full = [(a, b, c) for a in one for b in one for c in one]
    if points == 27:
        return full
    if points == 7:
        return [o for o in full if sum(map(abs, o)) <= 1]
    flat = [o for o in full if o[2] == 0]
    return flat if points == 9 else [o for o in flat if sum(map(abs, o)) <= 1]


def _stencil(case, g, dtype, jitter=1e-3):
    """(rows, columns, values) of a stencil matrix, sorted by row and column."""
    ni, nj, nk, offs = case["ni"], case["nj"], case["nk"], _offsets(case["points"])
    n = ni * nj * nk
    at = torch.arange(n, device=DEVICE, dtype=torch.int32)
    i, j, k = at // (nj * nk), (at // nk) % nj, at % nk
    keep = torch.stack([(i + a >= 0) & (i + a < ni) & (j + b >= 0) & (j + b < nj) & (k + c >= 0) & (k + c < nk)
                        for a, b, c in offs], 1)
    step = torch.tensor([a * nj * nk + b * nk + c for a, b, c in offs], device=DEVICE, dtype=torch.int32)
    centre = torch.tensor([float(len(offs) - 1) if o == (0, 0, 0) else -1.0 for o in offs], device=DEVICE, dtype=dtype)
    cols = (at[:, None] + step[None, :])[keep]
    rows = at[:, None].expand(-1, len(offs))[keep]
    vals = centre[None, :].expand(n, -1)[keep]
    if jitter:
        vals = vals + jitter * torch.randn(vals.numel(), generator=g, device=DEVICE, dtype=dtype)
    extra = int(round(case.get("offband", 0.0) * rows.numel()))
    if not extra:
        return n, rows, cols, vals
    key = rows.long() * n + cols
    new = torch.unique(torch.randint(0, n * n, (2 * extra + 64,), generator=g, device=DEVICE))
    found = torch.searchsorted(key, new).clamp_(max=key.numel() - 1)
    new = new[key[found] != new]
    new = new[torch.randperm(new.numel(), generator=g, device=DEVICE)[:extra]]
    key, order = torch.cat([key, new]).sort()
    vals = torch.cat([vals, _normal(g, new.numel(), dtype)])[order]
    return n, (key // n).int(), (key % n).int(), vals


def _random_columns(lens, limit, g):
    """(rows, columns) of rows with the given lengths: sorted distinct random columns below each row's limit."""
    rows = torch.repeat_interleave(torch.arange(lens.numel(), device=DEVICE), lens)
    room = (limit - lens + 1)[rows]
    wide = int(limit.max()) + 1
    draws = (torch.rand(rows.numel(), generator=g, device=DEVICE, dtype=torch.float64) * room).long()
    draws = torch.sort(rows * wide + draws)[0] - rows * wide
    first = torch.cumsum(lens, 0) - lens
    return rows.int(), (draws + torch.arange(rows.numel(), device=DEVICE) - first[rows]).int()


def _power_law(case, g, dtype):
    n = case["nrows"]
    # the same row lengths in another order for every seed, so that all have as many entries
    lens = torch.exp(MU + SIGMA * torch.randn(n, generator=_gen(1), device=DEVICE)).round_().clamp_(1, min(MAX_ROW, n))
    lens = lens.long()[torch.randperm(n, generator=g, device=DEVICE)]
    rows, cols = _random_columns(lens, torch.full_like(lens, n), g)
    return n, rows, cols, _normal(g, rows.numel(), dtype)


def _triplets(case, g):
    build = _stencil if case["structure"] == "stencil" else _power_law
    return build(case, g, DTYPES[case["dtype"]])


def _coo(n, rows, cols, vals):
    return CooMatrix(n, n, vals.numel(), rows, cols, vals, dtype=vals.dtype, device=DEVICE)


def _csr(n, rows, cols, vals):
    ro = torch.zeros(n + 1, dtype=torch.int32, device=DEVICE)
    ro[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return CsrMatrix(n, n, vals.numel(), ro, cols, vals, dtype=vals.dtype, device=DEVICE)


def _laplacian(case):
    """The 5-point Laplacian (4 and -1)."""
    grid = {"ni": case["ni"], "nj": case["nj"], "nk": 1, "points": 5}
    return _stencil(grid, None, DTYPES[case["dtype"]], jitter=0.0)


def _batch_parts(case, g):
    """Sizes, and one CSR over all the batch's matrices with columns counted from each one's own start."""
    count, dtype, fixed = case["count"], DTYPES[case["dtype"]], _gen(2)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    spread = torch.rand(count, generator=fixed, device=DEVICE, dtype=torch.float64)
    size = torch.exp(spread * (hi - lo) + lo).round().long()
    lam = torch.rand(count, generator=fixed, device=DEVICE) * (LAM_HI - LAM_LO) + LAM_LO
    own = torch.repeat_interleave(torch.arange(count, device=DEVICE), size)  # the matrix of each row
    lens = torch.minimum(torch.poisson(lam[own], generator=fixed).long(), size[own])
    rows, cols = _random_columns(lens, size[own], g)
    ro = torch.zeros(own.numel() + 1, dtype=torch.int64, device=DEVICE)
    ro[1:] = torch.cumsum(lens, 0)
    vals = _normal(g, rows.numel(), dtype)
    x = _uniform(g, own.numel(), dtype)
    return size, own, rows, ro, cols, vals, x


def _prepare_batch(case, g):
    size, _, _, ro, cols, vals, x = _batch_parts(case, g)
    first = torch.zeros(size.numel() + 1, dtype=torch.int64, device=DEVICE)
    first[1:] = torch.cumsum(size, 0)
    row0, ent0 = first.tolist(), ro[first].tolist()
    y = torch.zeros_like(x)
    mats, xs, ys = [], [], []
    for m in range(size.numel()):
        a, b, s, t = row0[m], row0[m + 1], ent0[m], ent0[m + 1]
        mats.append(CsrMatrix(b - a, b - a, t - s, (ro[a:b + 1] - s).int(), cols[s:t].clone(), vals[s:t].clone(),
                              dtype=vals.dtype, device=DEVICE))
        xs.append(x[a:b].clone())
        ys.append(y[a:b])
    batch = batched.CsrBatch(mats, xs, ys)
    batch.autotune()
    return {"case": case, "batch": batch, "y": y}


def prepare(case, seed):
    g, op = _gen(seed), case["op"]
    if op == "batch":
        return _prepare_batch(case, g)
    state = {"case": case}
    if op == "vectors":
        n, dtype = case["n"], DTYPES[case["dtype"]]
        state["x"] = _uniform(g, n, dtype)
        state["y"] = state["x"] * _uniform(g, n, dtype, 0.5, 1.5)
        state["z"] = _uniform(g, n, dtype, 0.0, 1.0)
        state["w"] = torch.empty_like(state["x"])
        return state
    if op == "cg":
        n, rows, cols, vals = _laplacian(case)
        state["A"] = _csr(n, rows, cols, vals)
        state["b"] = _uniform(g, n, vals.dtype)
        state["x"] = torch.zeros_like(state["b"])
        return state
    n, rows, cols, vals = _triplets(case, g)
    if op in ("assemble", "sort"):
        order = torch.randperm(vals.numel(), generator=g, device=DEVICE)
        state["A"] = _coo(n, rows[order], cols[order], vals[order])
    elif op == "convert":
        state["A"] = _coo(n, rows, cols, vals)
    elif op == "switch" or case["format"] == "csr":
        state["A"] = _csr(n, rows, cols, vals)
    else:
        state["A"] = _coo(n, rows, cols, vals)
        if case["format"] != "coo":
            width = P90_ROW if case["format"] == "hyb" else 0
            state["A"] = from_coo(state["A"], FORMATS[case["format"]], hyb_width=width)
    if op == "multiply":
        state["x"] = _uniform(g, n, vals.dtype)
        state["y"] = _uniform(g, n, vals.dtype)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _arrays(A):
    """Every array of a container."""
    fmt = A.format_index()
    if fmt == COO_FORMAT:
        return {"rows": A.row_indices(), "columns": A.column_indices(), "values": A.values()}
    if fmt == CSR_FORMAT:
        return {"offsets": A.row_offsets(), "columns": A.column_indices(), "values": A.values()}
    if fmt == DIA_FORMAT:
        return {"offsets": A.diagonal_offsets(), "values": A.values_flat()}
    if fmt == ELL_FORMAT:
        return {"columns": A.column_indices().t(), "values": A.values().t()}
    if fmt == HYB_FORMAT:
        return {"ell": _arrays(A.ell()), "coo": _arrays(A.coo())}
    return {"dia": _arrays(A.dia()), "csr": _arrays(A.csr())}


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "multiply":
        multiply(state["A"], state["x"], state["y"], init=case["init"])
        return state["y"]
    if op == "vectors":
        n, x, y, w = case["n"], state["x"], state["y"], state["w"]
        waxpby(n, case["alpha"], x, case["beta"], y, w)
        return {"dot": dot(n, x, y), "sum": reduce(state["z"], n), "w": w}
    if op == "batch":
        state["batch"].multiply()
        return state["y"]
    if op == "cg":
        state["x"].zero_()
        iters, residual = solvers.cg(state["A"], state["b"], state["x"], max_iters=case["iters"], rtol=0.0)
        return {"x": state["x"], "iterations": iters, "residual": residual}
    if op == "assemble":
        return _arrays(convert(state["A"], CsrMatrix(dtype=state["A"].dtype, device=DEVICE)))
    if op == "sort":
        A = to_coo(state["A"])
        sort_by_row_and_column(A)
        return _arrays(A)
    if op == "convert":
        width = P90_ROW if case["format"] == "hyb" else 0
        return _arrays(from_coo(state["A"], FORMATS[case["format"]], hyb_width=width))
    A = DynamicMatrix(state["A"])
    status = convert(A, -1)
    return {"status": int(status), "format": A.active_index(), **_arrays(A.active())}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its outputs in 64 bits
# ---------------------------------------------------------------------------

def _sizes(case):
    """(rows, nonzeros) of the case's matrix: exact for stencils, the mean for random ones."""
    if case.get("structure") == "power_law":
        return case["nrows"], int(case["nrows"] * min(MEAN_ROW, case["nrows"]))
    ni, nj, nk, points = case["ni"], case["nj"], case.get("nk", 1), case.get("points", 5)
    n = ni * nj * nk
    if points == 27:
        z = (3 * ni - 2) * (3 * nj - 2) * (3 * nk - 2)
    elif points == 9:
        z = (3 * ni - 2) * (3 * nj - 2)
    else:
        z = points * n - 2 * sum(n // d for d in ((ni, nj, nk) if points == 7 else (ni, nj)))
    return n, z + int(round(case.get("offband", 0.0) * z))


def _matrix_bytes(case, fmt, n, z, size):
    """Bytes of the arrays; padding that holds no entry is not counted."""
    if fmt == "dia":
        return size * case["points"] * n
    if fmt == "hdc":
        off = z - z / (1 + case["offband"])
        return size * case["points"] * n + off * (4 + size) + 4 * n
    return z * (4 + size) + (4 * z if fmt == "coo" else 4 * n if fmt == "csr" else 0)


def work(case):
    op = case["op"]
    size = 8 if case["dtype"] == "f64" else 4
    if op == "vectors":
        return {"bytes": 6 * size * case["n"], "flops": 6 * case["n"]}
    if op == "batch":
        rows = case["count"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        z = rows * (LAM_LO + LAM_HI) / 2
        return {"bytes": z * (4 + size) + rows * (4 + 2 * size), "flops": 2 * z}
    n, z = _sizes(case)
    if op == "cg":
        # per iteration: the matrix, p read and Ap written; x, r, p and Ap read, x, r and p written
        return {"bytes": case["iters"] * (z * (4 + size) + 4 * n + 9 * size * n),
                "flops": case["iters"] * (2 * z + 10 * n)}
    if op in ("assemble", "sort", "convert"):
        out = {"assemble": "csr", "sort": "coo"}.get(op) or case["format"]
        return {"bytes": z * (8 + size) + _matrix_bytes(case, out, n, z, size), "flops": 0}
    if op == "switch":
        out = "dia" if case["structure"] == "stencil" else "csr"
        return {"bytes": _matrix_bytes(case, "csr", n, z, size) + (_matrix_bytes(case, "dia", n, z, size)
                                                                   if out == "dia" else 0), "flops": 0}
    return {"bytes": _matrix_bytes(case, case["format"], n, z, size) + size * n * (2 if case["init"] else 3),
            "flops": 2 * z}


def _product(n, rows, cols, vals, x):
    y = torch.zeros(n, dtype=torch.float64, device=DEVICE)
    for a in range(0, vals.numel(), 1 << 25):
        b = a + (1 << 25)
        y.index_add_(0, rows[a:b], vals[a:b].double() * x[cols[a:b]].double())
    return y


def exact(case, seed):
    g, op = _gen(seed), case["op"]
    if op == "vectors":
        s = prepare(case, seed)
        x, y, z = s["x"].double(), s["y"].double(), s["z"].double()
        c = torch.tensor([case["alpha"], case["beta"]], dtype=DTYPES[case["dtype"]]).double().tolist()
        return {"dot": float((x * y).sum()), "sum": float(z.sum()), "w": c[0] * x + c[1] * y}
    if op == "batch":
        size, own, rows, _, cols, vals, x = _batch_parts(case, g)
        first = torch.cumsum(size, 0) - size
        return _product(x.numel(), rows, first[own[rows]] + cols, vals, x)
    if op == "cg":
        n, rows, cols, vals = _laplacian(case)
        b = _uniform(g, n, vals.dtype).double()
        grid = (case["ni"], case["nj"])

        def apply(v):
            v = v.view(grid)
            out = 4.0 * v
            out[1:] -= v[:-1]
            out[:-1] -= v[1:]
            out[:, 1:] -= v[:, :-1]
            out[:, :-1] -= v[:, 1:]
            return out.view(-1)

        x, r, p = torch.zeros_like(b), b.clone(), b.clone()
        rr = bb = float(r @ r)
        for _ in range(case["iters"]):
            ap = apply(p)
            alpha = rr / float(p @ ap)
            x += alpha * p
            r -= alpha * ap
            last, rr = rr, float(r @ r)
            p = r + (rr / last) * p
        return {"x": x, "iterations": None, "residual": math.sqrt(rr / bb)}
    if op != "multiply":
        return None  # indices and values that are moved, not computed
    n, rows, cols, vals = _triplets(case, g)
    x = _uniform(g, n, vals.dtype)
    y0 = _uniform(g, n, vals.dtype).double()
    y = _product(n, rows, cols, vals, x)
    return y if case["init"] else y0 + y
