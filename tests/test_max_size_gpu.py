"""Maximum sizes: a CSR matrix whose nnz sits just below the int32 limit the
kernels accept (2^31 - 4096), built on the device: every CSR kernel and the
COO kernel give the exact window sums (values 1, column j of row r is
(r + j) mod ncols), checked against an FP64 prefix-sum computation."""
import ctypes as C

import pytest
import torch

import morpheus_gb300 as mgb
from morpheus_gb300 import _lib

pytestmark = [pytest.mark.gpu, pytest.mark.slow]

L = 1000                       # entries per row
N = (2 ** 31 - 4096) // L - 1  # rows: nnz just under the limit
M = 3_000_001                  # columns


@pytest.fixture(scope="module")
def big(cuda):
    if torch.cuda.get_device_properties(0).total_memory < 80 * 2**30:
        pytest.skip("needs a GPU with >= 80 GB")
    dev = torch.device("cuda")
    nnz = N * L
    ro = (torch.arange(N + 1, device=dev, dtype=torch.int64) * L).to(torch.int32)
    r = torch.arange(N, device=dev, dtype=torch.int64)
    ci = torch.empty(nnz, dtype=torch.int32, device=dev)
    step = 1 << 14  # rows per piece, to bound the int64 temporaries
    j = torch.arange(L, device=dev, dtype=torch.int64)
    for a in range(0, N, step):
        b = min(N, a + step)
        ci[a * L:b * L] = ((r[a:b, None] + j[None, :]) % M).reshape(-1).to(torch.int32)
    va = torch.ones(nnz, dtype=torch.float64, device=dev)
    x = torch.rand(M, dtype=torch.float64, device=dev, generator=torch.Generator(device=dev).manual_seed(5)) - 0.5
    # y_ref[r] = sum_{j<L} x[(r + j) mod M] from an FP64 prefix sum of x repeated
    xx = torch.cat([x, x[:L]])
    cs = torch.cat([torch.zeros(1, dtype=torch.float64, device=dev), torch.cumsum(xx, 0)])
    rm = r % M
    y_ref = cs[rm + L] - cs[rm]
    A = mgb.CsrMatrix(N, M, nnz, ro, ci, va)
    yield A, x, y_ref
    del A, ci, va


@pytest.mark.parametrize("variant", [mgb.CSR_SEGMENTS, mgb.CSR_ROWS, mgb.CSR_SPLIT, mgb.CSR_ROWS_GATHER])
def test_csr_at_int32_limit(big, variant):
    A, x, y_ref = big
    A._variant = variant
    y = torch.empty(N, dtype=torch.float64, device="cuda")
    mgb.multiply(A, x, y)
    torch.cuda.synchronize()
    err = (torch.linalg.norm(y - y_ref) / torch.linalg.norm(y_ref)).item()
    assert err <= 1e-12, err


def test_chooser_and_coo_at_int32_limit(big):
    A, x, y_ref = big
    A.forget_kernel_variant()
    assert A.kernel_variant() == mgb.CSR_SPLIT  # rows of 1000 entries on average
    coo = mgb.to_coo(A)
    y = torch.empty(N, dtype=torch.float64, device="cuda")
    mgb.multiply(coo, x, y)
    torch.cuda.synchronize()
    err = (torch.linalg.norm(y - y_ref) / torch.linalg.norm(y_ref)).item()
    assert err <= 1e-12, err


# More rows than 2^30, three entries in every 128 of them: the sum of two row
# numbers passes 2^31.  Values and x are small integers, so row sums are exact.
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("planned", [True, False])
def test_csr_beyond_2_30_rows(cuda, planned, dtype):
    if torch.cuda.get_device_properties(0).total_memory < 120 * 2**30:
        pytest.skip("needs a GPU with >= 120 GB")
    dev, rows, ncols = torch.device("cuda"), (1 << 30) + (1 << 20) + 77, 1009
    groups = rows // 128 + 1
    r = torch.arange(rows + 1, device=dev, dtype=torch.int64)
    ro = (r // 128 * 3 + (r % 128 > 3).int() + 2 * (r % 128 > 70).int()).to(torch.int32)
    del r
    nnz = int(ro[-1])
    ci = (torch.arange(nnz, device=dev, dtype=torch.int64) * 7919 % ncols).to(torch.int32)
    x = torch.arange(ncols, device=dev).to(dtype) - 500
    A = mgb.CsrMatrix(rows, ncols, nnz, ro, ci, torch.ones(nnz, dtype=dtype, device=dev), dtype=dtype)
    want = torch.zeros(groups * 128, dtype=dtype, device=dev)
    xv = torch.cat([x[ci.long()], torch.zeros(3, dtype=dtype, device=dev)])
    first = torch.arange(groups, device=dev, dtype=torch.int64) * 3
    want[3::128] = xv[first.clamp(max=nnz)]
    want[70::128] = xv[(first + 1).clamp(max=nnz)] + xv[(first + 2).clamp(max=nnz)]
    want = want[:rows]
    y = torch.full((rows,), 7, dtype=dtype, device=dev)
    if planned:
        A._variant = mgb.CSR_SEGMENTS
        mgb.multiply(A, x, y)
    else:
        desc, name = A._desc(), "mgb_spmv_csr_" + ("f64" if dtype == torch.float64 else "f32")
        _lib.call(name, C.byref(desc), x.data_ptr(), y.data_ptr(), 1, None)
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_coo_of_2_31_rows(cuda):
    """The largest number of rows (2^31 - 1), an entry in every 65,536: rows are zero-filled up to the last one."""
    if torch.cuda.get_device_properties(0).total_memory < 80 * 2**30:
        pytest.skip("needs a GPU with >= 80 GB")
    dev, rows = torch.device("cuda"), (1 << 31) - 1
    ri = torch.arange(0, rows, 65536, device=dev, dtype=torch.int64)
    A = mgb.CooMatrix(rows, 3, ri.numel(), ri.int(), torch.ones_like(ri).int(),
                      torch.full((ri.numel(),), 2.0, dtype=torch.float32, device=dev), dtype=torch.float32)
    x = torch.tensor([0.0, 3.0, 0.0], device=dev)
    y = torch.full((rows,), 7.0, dtype=torch.float32, device=dev)
    mgb.multiply(A, x, y)
    torch.cuda.synchronize()
    assert torch.all(y[ri] == 6.0) and int(torch.count_nonzero(y)) == ri.numel()
