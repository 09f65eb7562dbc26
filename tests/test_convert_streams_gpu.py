"""GPU: conversions on a stream of the caller's, beside work on the current one."""
import numpy as np
import pytest
import torch

import morpheus_gb300 as mgb
from helpers import assert_same_matrix
from morpheus_gb300 import generators as gen
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(fmt, shuffled):
    hm = gen.csr_to_coo_host(gen.stencil_27pt(24, seed=fmt))
    if shuffled:
        p = np.random.default_rng(fmt).permutation(hm["nnz"])
        hm = dict(hm, row_indices=hm["row_indices"][p], column_indices=hm["column_indices"][p], values=hm["values"][p])
    return hm


def _late_writes():
    """Blocks of many sizes, filled by kernels that wait behind a long one on the current stream, then dropped: their
    memory is free for the current stream's next tensors and still to be written."""
    torch.cuda.empty_cache()
    blocks = [torch.empty(1 << k, dtype=torch.uint8, device="cuda") for k in range(9, 25) for _ in range(4)]
    a = torch.full((8192, 8192), 1e-4, device="cuda")
    for _ in range(8):
        a = a @ a
    for b in blocks:
        b.fill_(255)


@pytest.mark.parametrize("handle", [False, True])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("fmt", [1, 2, 3, 4, 5])
def test_conversion_beside_the_current_stream(cuda, fmt, shuffled, handle):
    hm = _case(fmt, shuffled)
    A = mgb.matrix_from_host(hm)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    _late_writes()
    out = mgb.from_coo(A, fmt, stream=side.cuda_stream if handle else side)
    torch.cuda.synchronize()
    assert_same_matrix(mgb.matrix_to_host(out), O.OracleMatrix.from_host(hm).convert(fmt).to_host())


@pytest.mark.parametrize("fmt", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("unsorted", [False, True])
def test_switch_in_place_beside_the_current_stream(cuda, fmt, unsorted):
    """CSR -> fmt; with rows out of order the entries take the way through a COO temporary."""
    A = gen.stencil_27pt(24, seed=1)
    if unsorted:
        s = slice(A["row_offsets"][50], A["row_offsets"][51])
        A["column_indices"][s] = A["column_indices"][s][::-1].copy()
    dyn, side = mgb.DynamicMatrix(mgb.matrix_from_host(A)), torch.cuda.Stream()
    torch.cuda.synchronize()
    _late_writes()
    assert mgb.convert(dyn, fmt, stream=side) == mgb.conversion_error_e.CONV_SUCCESS
    _late_writes()  # what the conversion dropped is not handed out while it still reads it
    torch.cuda.synchronize()
    assert_same_matrix(mgb.matrix_to_host(dyn.active()), O.OracleMatrix.from_host(A).convert(fmt).to_host())


def test_sort_beside_the_current_stream(cuda):
    hm = _case(0, True)
    A, side = mgb.matrix_from_host(hm), torch.cuda.Stream()
    torch.cuda.synchronize()
    _late_writes()
    mgb.sort_by_row_and_column(A, stream=side)
    torch.cuda.synchronize()
    om = O.OracleMatrix.from_host(hm)
    om.sort_by_row_and_column()
    assert_same_matrix(mgb.matrix_to_host(A), om.to_host())


@pytest.mark.parametrize("fmt", [1, 2, 3, 4, 5])
def test_results_are_allocated_on_the_stream(cuda, fmt):
    A, side = mgb.matrix_from_host(_case(fmt, False)), torch.cuda.Stream()
    torch.cuda.synchronize()
    out = mgb.from_coo(A, fmt, stream=side)
    torch.cuda.synchronize()
    B = out.ell() if fmt == 4 else out.dia() if fmt == 5 else out
    at = (B.values_flat() if hasattr(B, "values_flat") else B.values()).data_ptr()
    streams = [s["stream"] for s in torch.cuda.memory_snapshot()
               if s["address"] <= at < s["address"] + s["total_size"]]
    assert streams == [side.cuda_stream]


def test_default_stream_by_its_handle(cuda):
    hm = _case(2, False)
    A, side = mgb.matrix_from_host(hm), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        out = mgb.from_coo(A, 2, stream=0)
    torch.cuda.synchronize()
    assert_same_matrix(mgb.matrix_to_host(out), O.OracleMatrix.from_host(hm).convert(2).to_host())
