"""GPU conversions at the edges of their tiles: every result bit-identical to the oracle's Serial convert."""
import numpy as np
import pytest

from morpheus_gb300 import generators as gen
from test_convert_gpu import check_all_targets, both
from helpers import assert_same_matrix
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def diagonals(N, M, nd, seed, dtype, keep=0.7):
    """Sorted COO with entries on nd random diagonals (each slot present with probability `keep`)."""
    rng = np.random.default_rng(seed)
    offs = np.sort(rng.choice(np.arange(-(N - 1), M), nd, replace=False))
    r = np.arange(N)[:, None]
    c = r + offs[None, :]
    m = (c >= 0) & (c < M) & (rng.random((N, nd)) < keep)
    rows, cols = np.broadcast_to(r, c.shape)[m], c[m]
    return {"format": 0, "nrows": N, "ncols": M, "nnz": rows.size, "row_indices": rows.astype(np.int32),
            "column_indices": cols.astype(np.int32), "values": rng.standard_normal(rows.size).astype(dtype)}


# one diagonal; 512-row tiles; the last size whose diagonals fit one tile and the first that needs 32 rows or
# several groups of diagonals; the lookup table's limit (256); more groups than the tiles take
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,nd", [(1, 1), (33, 3), (1025, 7), (513, 8), (700, 63), (640, 124), (611, 125), (500, 256),
                                  (501, 257), (900, 700), (1500, 2100), (2301, 4200)])
def test_dia_tiles(cuda, N, nd, dtype):
    hm = diagonals(N, N, min(nd, 2 * N - 1), seed=N + nd, dtype=dtype, keep=0.7 if nd < 1000 else 0.1)
    got, ref = both(hm, O.DIA)
    assert_same_matrix(got, ref)


@pytest.mark.parametrize("N,M", [(97, 400), (400, 97)])
def test_dia_tiles_nonsquare(cuda, N, M):
    got, ref = both(diagonals(N, M, 40, seed=N, dtype=np.float64), O.DIA)
    assert_same_matrix(got, ref)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("gap", [1, 255, 256, 257, 3000])
def test_row_starts_over_gaps(cuda, gap, shift):
    """Empty rows before, between (around the gap that a CTA fills together) and after the entries; entries from
    an offset in their arrays that 16-byte loads do not allow."""
    rng = np.random.default_rng(gap)
    rows = np.repeat(np.arange(7, 7 + 40 * (gap + 1), gap + 1), rng.integers(1, 9, 40))
    n = rows.size
    N = int(rows[-1]) + 1 + 2 * gap
    cols = np.concatenate([np.sort(rng.choice(N, int((rows == r).sum()), replace=False)) for r in np.unique(rows)])
    hm = {"format": 0, "nrows": N, "ncols": N, "nnz": n, "row_indices": rows.astype(np.int32),
          "column_indices": cols.astype(np.int32), "values": rng.standard_normal(n)}
    if not shift:
        check_all_targets(hm)
        return
    import torch

    import morpheus_gb300 as mgb
    A = mgb.CooMatrix(N, N, n, *(torch.from_numpy(np.concatenate([a[:1], a])).cuda()[1:] for a in (
        hm["row_indices"], hm["column_indices"], hm["values"])))
    for fmt in (1, 2, 3, 4, 5):
        want = O.OracleMatrix.from_host(hm).convert(fmt).to_host()
        assert_same_matrix(mgb.matrix_to_host(mgb.from_coo(A, fmt)), want)


# gaps that are listed: more than a CTA's list holds, around the length from which the whole grid fills them, both kinds
@pytest.mark.parametrize("gaps", [[258] * 2100, [65535, 65536, 65537, 65538], [65537] * 3 + [257, 300000, 1, 256] * 2,
                                  [1] * 1023 + [70000] + [1] * 1024 + [5000]])
def test_row_starts_over_long_gaps(cuda, gaps):
    rng = np.random.default_rng(len(gaps))
    rows = 3 + np.cumsum(np.asarray([0] + gaps))
    rows = np.repeat(rows, rng.integers(1, 3, rows.size))
    n, N = rows.size, int(rows[-1]) + 5
    order = np.lexsort((np.arange(n) % 2, rows))
    hm = {"format": 0, "nrows": N, "ncols": 7, "nnz": n, "row_indices": rows.astype(np.int32),
          "column_indices": (np.arange(n)[order] % 2 + 1).astype(np.int32), "values": rng.standard_normal(n)}
    for fmt in (O.CSR, O.ELL, O.HYB):
        got, ref = both(hm, fmt)
        assert_same_matrix(got, ref, f"{fmt}:")


def test_stencil_tiles(cuda):
    check_all_targets(gen.stencil_27pt(23, seed=5))


# rows of a staged tile's limits (32 x 64 entries), even lengths, a row beyond the staging, a slab wider than the rows
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,lens,width", [(1, [3], 0), (257, [5], 4), (300, [16, 32], 0), (65, [64], 40),
                                          (100, [63, 65], 33), (70, [0, 2500, 1, 0], 7), (511, [0, 1, 2], 1)])
def test_ell_and_hyb_tiles(cuda, N, lens, width, dtype):
    A = gen.random_lengths_csr(N, 4000, np.resize(np.asarray(lens), N), seed=N, dtype=dtype)
    coo = gen.csr_to_coo_host(A)
    for fmt, w in ((O.ELL, 0), (O.HYB, 0), (O.HYB, width)):
        got, ref = both(coo, fmt, hyb_width=w)
        assert_same_matrix(got, ref, f"{fmt} width {w}:")


# slabs too wide for their rows: several segments of the slot columns, rows beyond the staging (whole blocks of their
# slots, a last block that is not full), one long row among short ones
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,lens,width", [(1, [70000], 0), (33, [9001, 8990, 9008], 0), (64, [5000], 4999),
                                          (300, [3] * 299 + [12345], 700), (257, [2] * 100 + [4097] + [7] * 156, 64)])
def test_wide_slabs(cuda, N, lens, width, dtype):
    A = gen.random_lengths_csr(N, 80000, np.resize(np.asarray(lens), N), seed=N, dtype=dtype)
    coo = gen.csr_to_coo_host(A)
    for fmt, w in ((O.ELL, 0), (O.HYB, 0), (O.HYB, width)):
        got, ref = both(coo, fmt, hyb_width=w)
        assert_same_matrix(got, ref, f"{fmt} width {w}:")


# rows whose entries past the ELL width are at the limit of a warp's copy (4,096), several pieces, the whole COO part
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("lens,width", [([4095 + 5], 5), ([4096 + 5, 3], 5), ([1, 30000, 0, 9, 4101], 5), ([40960 + 1], 1),
                                        ([2040] * 3 + [4096] + [4097] * 2, 1), ([6, 9, 4], 4)])
def test_hyb_long_rows(cuda, lens, width, dtype):
    A = gen.random_lengths_csr(len(lens), 50000, np.asarray(lens), seed=width, dtype=dtype)
    got, ref = both(gen.csr_to_coo_host(A), O.HYB, hyb_width=width)
    assert_same_matrix(got, ref)


# all, some or none of the entries on true diagonals; more true diagonals than the lookup table takes
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,nd,keep", [(3, 3, 1.0), (64, 5, 0.9), (513, 40, 0.6), (700, 500, 0.5), (1200, 1500, 0.4),
                                       (400, 300, 0.1)])
def test_hdc_tiles(cuda, N, nd, keep, dtype):
    got, ref = both(diagonals(N, N, nd, seed=nd, dtype=dtype, keep=keep), O.HDC)
    assert_same_matrix(got, ref)


# rows with more entries off the diagonals than a warp walks or compacts itself (512 or 4,096; pieces of 2,048; 2,048 per
# 32 diagonals): first, last, neighbouring, beside short and empty rows
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nd", [1, 3, 40, 300])
@pytest.mark.parametrize("rows,length", [([0], 513), ([5999], 6000), ([31, 32, 33], 2100), ([100, 101, 4000], 5000),
                                         (list(range(64, 128)), 4096)])
def test_hdc_long_rows(cuda, rows, length, nd, dtype):
    N = 6000
    rng = np.random.default_rng(nd + length)
    hm = diagonals(N, N, nd, seed=nd, dtype=dtype, keep=1.0)
    if nd == 3:  # offsets near the middle: every diagonal is a long one
        r = np.arange(1, N - 1)
        key = np.unique(np.concatenate([r * N + r + d for d in (-1, 0, 1)]))
    else:
        key = hm["row_indices"].astype(np.int64) * N + hm["column_indices"]
    key = np.unique(np.concatenate([key] + [r * N + np.sort(rng.choice(N, length, replace=False)) for r in rows]))
    key = key[(key // N != 34) & (key // N != 4001)]  # empty rows
    hm = {"format": 0, "nrows": N, "ncols": N, "nnz": key.size, "row_indices": (key // N).astype(np.int32),
          "column_indices": (key % N).astype(np.int32), "values": rng.standard_normal(key.size).astype(dtype)}
    got, ref = both(hm, O.HDC)
    assert_same_matrix(got, ref)


def _two_call(A, fmt, like):
    """The conversion through its own *_plan and fill entry points, into a container of `like`'s sizes."""
    import ctypes as C

    import morpheus_gb300 as mgb
    from morpheus_gb300 import _lib
    from morpheus_gb300.convert import _new_coo, _new_csr, _new_dia, _new_ell
    name = {2: "dia", 3: "ell", 4: "hyb", 5: "hdc"}[fmt]
    sd, sizes = A._desc(), [C.c_int64() for _ in range(1 if fmt < 4 else 3)]
    more = [0] if fmt == 4 else []
    _lib.call(f"mgb_convert_coo_to_{name}_plan", C.byref(sd), *more, *[C.byref(z) for z in sizes], None)
    n, m, z, dt, dev = A.nrows(), A.ncols(), A.nnnz(), A.dtype, A.device
    s = [v.value for v in sizes]
    out = {2: lambda: _new_dia(n, m, z, s[0], dt, dev), 3: lambda: _new_ell(n, m, z, s[0], dt, dev),
           4: lambda: mgb.HybMatrix(_new_ell(n, m, s[1], s[0], dt, dev), _new_coo(n, m, s[2], dt, dev), dt, dev),
           5: lambda: mgb.HdcMatrix(_new_dia(n, m, s[1], s[0], dt, dev), _new_csr(n, m, s[2], dt, dev), dt, dev)}[fmt]()
    dd = out._desc()
    _lib.call(f"mgb_convert_coo_to_{name}_f64", C.byref(sd), C.byref(dd), None)
    return mgb.matrix_to_host(out)


@pytest.mark.parametrize("fmt", [2, 3, 4, 5])
@pytest.mark.parametrize("shuffled", [False, True])
def test_planned_conversion_equals_separate_calls(cuda, fmt, shuffled):
    import torch

    import morpheus_gb300 as mgb
    hm = diagonals(301, 301, 60, seed=fmt, dtype=np.float64)
    if shuffled:
        p = np.random.default_rng(1).permutation(hm["nnz"])
        hm = dict(hm, row_indices=hm["row_indices"][p], column_indices=hm["column_indices"][p], values=hm["values"][p])
    A = mgb.matrix_from_host(hm)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    planned = mgb.from_coo(A, fmt, stream=side)
    side.synchronize()
    got = mgb.matrix_to_host(planned)
    assert_same_matrix(got, _two_call(A, fmt, planned))
    assert_same_matrix(got, O.OracleMatrix.from_host(hm).convert(fmt).to_host())


# rows at the limits of the sorted tiles (512), of a tile's window (1024), of the shared-memory sort (4096) and of its
# merge passes; many empty rows; a few rows that hold everything
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,lens", [(1, [1]), (5, [0, 7, 0]), (900, [1, 2, 31, 32, 33]), (40, [511, 512, 513, 3]),
                                    (12, [1023, 1, 1024, 600, 600]), (5, [4096, 4097, 0, 2]), (3, [20000, 5]),
                                    (60000, [1] + [0] * 99)])
def test_row_sort_tiles(cuda, N, lens, dtype):
    import torch

    import morpheus_gb300 as mgb
    rng = np.random.default_rng(N)
    rows = np.repeat(np.arange(N), np.resize(np.asarray(lens), N))
    cols = rng.integers(0, 3000, rows.size)  # duplicates among them
    p = rng.permutation(rows.size)
    hm = {"format": 0, "nrows": N, "ncols": 3000, "nnz": rows.size, "row_indices": rows[p].astype(np.int32),
          "column_indices": cols.astype(np.int32), "values": rng.standard_normal(rows.size).astype(dtype)}
    got, ref = both(hm, O.CSR)
    assert_same_matrix(got, ref)
    om = O.OracleMatrix.from_host(hm)
    om.sort_by_row_and_column()
    A = mgb.matrix_from_host(hm)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    mgb.sort_by_row_and_column(A, stream=side)
    side.synchronize()
    assert_same_matrix(mgb.matrix_to_host(A), om.to_host())


# rows that several CTAs sort in pieces (4,096): one entry past a piece, full pieces, odd and even numbers of merge levels,
# a last run without a neighbour, rows of different levels together; many equal columns
@pytest.mark.parametrize("ncols", [50, 1 << 20])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("lens", [[4097], [8192], [8193, 0, 3], [12289, 40000, 600, 4096], [70001, 2, 16384, 16385]])
def test_row_sort_pieces(cuda, lens, ncols, dtype):
    import morpheus_gb300 as mgb
    rng = np.random.default_rng(len(lens))
    rows = rng.permutation(np.repeat(np.arange(len(lens), dtype=np.int32), lens))
    cols = rng.integers(0, ncols, rows.size).astype(np.int32)
    hm = {"format": 0, "nrows": len(lens), "ncols": ncols, "nnz": rows.size, "row_indices": rows,
          "column_indices": cols, "values": rng.standard_normal(rows.size).astype(dtype)}
    got, ref = both(hm, O.CSR)
    assert_same_matrix(got, ref)
    A = mgb.matrix_from_host(hm)
    mgb.sort_by_row_and_column(A)
    om = O.OracleMatrix.from_host(hm)
    om.sort_by_row_and_column()
    assert_same_matrix(mgb.matrix_to_host(A), om.to_host())


# more records than L2 holds: scattered in two halves (the middle row on either side, an odd number of rows) or, with
# rows near each other, at once
@pytest.mark.parametrize("N", [4098, 65537])
@pytest.mark.parametrize("shuffled", [True, False])
def test_row_sort_beyond_l2(cuda, N, shuffled):
    import torch

    import morpheus_gb300 as mgb
    n = (1 << 23) + 77
    rng = np.random.default_rng(N)
    rows = rng.integers(0, N, n, dtype=np.int32)
    if not shuffled:
        rows.sort()
    cols = rng.integers(0, 1 << 20, n, dtype=np.int32)
    vals = np.arange(n, dtype=np.float32)
    order = np.lexsort((cols, rows))
    dev = [torch.from_numpy(a.copy()).cuda() for a in (rows, cols, vals)]
    A = mgb.CooMatrix(N, 1 << 20, n, *dev, dtype=torch.float32, device="cuda")
    mgb.sort_by_row_and_column(A)
    got = mgb.matrix_to_host(A)
    np.testing.assert_array_equal(got["row_indices"], rows[order])
    np.testing.assert_array_equal(got["column_indices"], cols[order])
    np.testing.assert_array_equal(got["values"], vals[order])


def _csr_host(coo):
    ro = np.zeros(coo["nrows"] + 1, np.int32)
    np.cumsum(np.bincount(coo["row_indices"], minlength=coo["nrows"]), out=ro[1:])
    return {"format": 1, "nrows": coo["nrows"], "ncols": coo["ncols"], "nnz": coo["nnz"], "row_offsets": ro,
            "column_indices": coo["column_indices"], "values": coo["values"]}


# the entries of a CSR matrix without its row indices: empty rows, rows longer than the 1,024 entries that a warp marks
# at a time, other shapes; and what goes through COO instead (columns out of order, repeated, non-square HDC)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("fmt", [2, 3, 4, 5])
@pytest.mark.parametrize("case", ["diagonals", "long", "empty_rows", "wide", "unsorted", "repeated"])
def test_csr_without_row_indices(cuda, case, fmt, dtype):
    import morpheus_gb300 as mgb
    rng = np.random.default_rng(7)
    if case == "diagonals":
        A = _csr_host(diagonals(777, 777, 90, seed=3, dtype=dtype))
    elif case == "long":
        A = gen.random_lengths_csr(70, 3000, np.resize([2, 2900, 0, 1023, 1025, 1], 70), seed=4, dtype=dtype)
    elif case == "empty_rows":
        A = gen.random_csr(3001, 3001, 0.0004, seed=5, dtype=dtype, empty_row_frac=0.5)
    elif case == "wide":
        A = gen.random_csr(301, 900, 0.02, seed=6, dtype=dtype)
    else:
        A = gen.random_csr(200, 200, 0.05, seed=8, dtype=dtype)
        cols, ro = A["column_indices"].copy(), A["row_offsets"]
        for r in np.flatnonzero(np.diff(ro) > 1)[::3]:
            if case == "unsorted":
                cols[ro[r]:ro[r + 1]] = cols[ro[r]:ro[r + 1]][::-1]
            else:
                cols[ro[r] + 1] = cols[ro[r]]
        A["column_indices"] = cols
    om = O.OracleMatrix.from_host(A)
    dyn = mgb.DynamicMatrix(mgb.matrix_from_host(A))
    status = mgb.convert(dyn, fmt)
    try:
        want = om.convert(fmt).to_host()
    except O.OracleError:
        assert status == mgb.conversion_error_e.PROXY_TO_DYNAMIC and dyn.active_index() == 1
        return
    assert status == mgb.conversion_error_e.CONV_SUCCESS
    assert_same_matrix(mgb.matrix_to_host(dyn.active()), want)


# rows that a warp leaves to other CTAs: 32 rows at the limit (8,192 entries) and past it, rows at the length limit (512),
# at a piece's end (2,048) and past it, among short and empty rows; entries out of order or equal across a piece's border
@pytest.mark.parametrize("fmt", [2, 3, 4, 5])
@pytest.mark.parametrize("case", ["in_order", "unsorted", "repeated", "outside"])
@pytest.mark.parametrize("lens", [[8192], [8193], [512] * 15 + [513], [512] * 16 + [513] * 16,
                                  [2, 4096, 4097, 0, 33], [8900] + [7] * 70 + [513]])
def test_csr_long_rows(cuda, lens, case, fmt):
    import morpheus_gb300 as mgb
    A = gen.random_lengths_csr(len(lens), 9000, np.asarray(lens), seed=fmt, dtype=np.float64)
    cols, r = A["column_indices"].copy(), int(np.argmax(lens))
    b = A["row_offsets"][r] + (2048 if lens[r] > 2048 else lens[r] // 2)
    if case == "unsorted":
        cols[b - 1:b + 1] = cols[b - 1:b + 1][::-1]
    elif case == "repeated":
        cols[b] = cols[b - 1]
    elif case == "outside":
        cols[A["row_offsets"][r + 1] - 1] = 9000
    A["column_indices"] = cols
    dyn = mgb.DynamicMatrix(mgb.matrix_from_host(A))
    status = mgb.convert(dyn, fmt)
    if case == "outside":
        assert status == mgb.conversion_error_e.PROXY_TO_DYNAMIC and dyn.active_index() == 1
        return
    try:
        want = O.OracleMatrix.from_host(A).convert(fmt).to_host()
    except O.OracleError:
        assert status == mgb.conversion_error_e.PROXY_TO_DYNAMIC
        return
    assert status == mgb.conversion_error_e.CONV_SUCCESS
    assert_same_matrix(mgb.matrix_to_host(dyn.active()), want)


def test_csr_with_offsets_that_do_not_span_its_entries(cuda):
    """Such a matrix converts as its COO form does."""
    import torch

    import morpheus_gb300 as mgb
    ro = torch.tensor([0, 2, 3, 3], dtype=torch.int32)
    A = mgb.CsrMatrix(3, 3, 5, ro, torch.tensor([0, 1, 2, 1, 2], dtype=torch.int32),
                      torch.arange(1, 6, dtype=torch.float64))
    for fmt in (2, 3, 4, 5):
        dyn = mgb.DynamicMatrix(A)
        assert mgb.convert(dyn, fmt) == mgb.conversion_error_e.CONV_SUCCESS
        assert_same_matrix(mgb.matrix_to_host(dyn.active()), mgb.matrix_to_host(mgb.from_coo(mgb.to_coo(A), fmt)))


# rows that a warp walks several at a time (32 / L of them) and counts by lane: every remainder of 32 / L, lengths at and
# past the warp's width, a change of length inside a warp's rows, a last warp that is not full; columns in order, with
# one row of a run out of order or with a column twice
@pytest.mark.parametrize("case", ["in_order", "unsorted", "repeated"])
@pytest.mark.parametrize("L", [3, 5, 9, 16, 17, 27, 31, 32, 33])
def test_csr_rows_of_equal_length(cuda, L, case):
    import morpheus_gb300 as mgb
    from morpheus_gb300 import analytics
    N = 32 * 9 + 19
    lens = np.full(N, L)
    lens[40], lens[100:132], lens[200:220] = 1, 0, max(1, L - 2)
    offs = np.array([d for k in range(17) for d in (-k, k + 1)][:L])
    ro = np.zeros(N + 1, np.int32)
    np.cumsum(lens, out=ro[1:])
    cols = np.concatenate([np.sort((r + offs[:lens[r]]) % N) for r in range(N)]).astype(np.int32)
    if case != "in_order":
        r = 32 * 5 + 11
        s = slice(ro[r], ro[r + 1])
        cols[s] = cols[s][::-1] if case == "unsorted" else np.r_[cols[s][0], cols[s][:-1]]
    A = {"format": 1, "nrows": N, "ncols": N, "nnz": cols.size, "row_offsets": ro, "column_indices": cols,
         "values": np.random.default_rng(L).standard_normal(cols.size)}
    om = O.OracleMatrix.from_host(A)
    M = mgb.matrix_from_host(A, device="cuda")
    assert np.array_equal(analytics.count_nnz_per_diagonal(M).cpu().numpy(), om.count_nnz_per_diagonal())
    for fmt in (O.DIA, O.HDC):
        dyn = mgb.DynamicMatrix(mgb.matrix_from_host(A, device="cuda"))
        status = mgb.convert(dyn, fmt)
        try:
            want = om.convert(fmt).to_host()
        except O.OracleError:
            assert status == mgb.conversion_error_e.PROXY_TO_DYNAMIC
            continue
        assert status == mgb.conversion_error_e.CONV_SUCCESS
        assert_same_matrix(mgb.matrix_to_host(dyn.active()), want)
