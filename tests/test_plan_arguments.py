"""Planned conversions refuse a plan that is not their source's, before anything is launched (no GPU needed)."""
import ctypes as C

import pytest

from morpheus_gb300 import _lib

BAD_ARGUMENT = 8
N, NNZ = 5000, 12000
AT = 1 << 20  # an address that nothing reads


def _plan(kind, fmt=2, sizes=(100, 0, 0), seen=0, n=N, nnz=NNZ):
    return _lib.CooPlan((C.c_int64 * 3)(*sizes), 0, fmt, seen, (C.c_int64 * 4)(kind, n, n, nnz), (C.c_void_p * 3)(AT, AT, AT))


def _call(name, src, plan):
    lib, dst = _lib.load(), _lib.Hdc()  # the largest container; its sizes agree with no plan
    more = (None, 0) if "_coo_" in name else ()
    return getattr(lib, name)(C.byref(src), C.byref(plan), C.byref(dst), *more, None)


CSR = _lib.Csr(N, N, NNZ, AT, AT, AT)
COO = _lib.Coo(N, N, NNZ, AT, AT, AT)
ROWS_DOWN, UNSORTED, DUPLICATE, BAD_OFFSETS = 2, 4, 8, 16


@pytest.mark.parametrize("dt", ["f64", "f32"])
@pytest.mark.parametrize("plan", [_plan(1), _plan(2, n=N + 1), _plan(2, nnz=NNZ - 1), _plan(2, seen=UNSORTED),
                                  _plan(2, seen=DUPLICATE), _plan(2, seen=BAD_OFFSETS), _plan(2, fmt=0),
                                  _plan(2, fmt=1), _plan(2, fmt=6), _plan(2, sizes=(257, 0, 0)), _plan(2, fmt=5, sizes=(745, 0, 0)),
                                  _plan(2, fmt=5, seen=UNSORTED)])
def test_csr_plan_of_another_source(lib_built, plan, dt):
    assert _call(f"mgb_convert_csr_planned_{dt}", CSR, plan) == BAD_ARGUMENT


def test_csr_plan_of_the_other_value_type(lib_built):
    """500 diagonals are 5 groups of an HDC's FP32 tiles and 9 of its FP64 ones: 6 are taken."""
    plan = _plan(2, fmt=5, sizes=(500, 0, 0))
    assert _call("mgb_convert_csr_planned_f64", CSR, plan) == BAD_ARGUMENT
    assert _call("mgb_convert_csr_planned_f32", CSR, plan) != BAD_ARGUMENT  # dst's sizes are refused later


def test_csr_plan_of_other_offsets(lib_built):
    other = _lib.Csr(N, N, NNZ, AT + 256, AT, AT)
    assert _call("mgb_convert_csr_planned_f64", other, _plan(2, sizes=(3, 0, 0))) == BAD_ARGUMENT


@pytest.mark.parametrize("dt", ["f64", "f32"])
@pytest.mark.parametrize("plan", [_plan(2), _plan(0), _plan(1, n=N - 1), _plan(1, nnz=NNZ + 1), _plan(1, fmt=0),
                                  _plan(1, fmt=6)])
def test_coo_plan_of_another_source(lib_built, plan, dt):
    assert _call(f"mgb_convert_coo_planned_{dt}", COO, plan) == BAD_ARGUMENT


def test_coo_without_row_indices(lib_built):
    src = _lib.Coo(N, N, NNZ, None, AT, AT)
    assert _call("mgb_convert_coo_planned_f64", src, _plan(1, seen=ROWS_DOWN)) == BAD_ARGUMENT
