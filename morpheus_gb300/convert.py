"""Format conversion on the device, with the reference's API:

    convert(src, dst)          Morpheus::convert<ExecSpace>(src, dst)
                               (core/src/Morpheus_Convert.hpp:53-57): dst's
                               format is the target; dst is resized and filled.
    convert(dyn, fmt) -> conversion_error_e
                               in-place switch of a DynamicMatrix through a
                               temporary COO (core/src/Morpheus_Convert.hpp:88-141);
                               on failure the matrix keeps its format and data.
    sort_by_row_and_column(coo), is_sorted(coo)
                               impl/Coo/Serial/Morpheus_Sort_Impl.hpp:109-186

All work runs in the CUDA kernels of convert.cu; results are bit-identical to
the reference's Serial conversions (including its tie-breaks and quirks).
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from .algorithms import _stream_handle, _suffix
from .containers import (COO_FORMAT, CSR_FORMAT, DIA_FORMAT, ELL_FORMAT, HDC_FORMAT, HYB_FORMAT, NFORMATS,
                         CooMatrix, CsrMatrix, DiaMatrix, DynamicMatrix, EllMatrix, HdcMatrix, HybMatrix,
                         _Matrix, _ptr, conversion_error_e, formats_e, get_pad_size)
from .exceptions import MorpheusException, NotImplementedException

_NAME = {COO_FORMAT: "coo", CSR_FORMAT: "csr", DIA_FORMAT: "dia", ELL_FORMAT: "ell", HYB_FORMAT: "hyb",
         HDC_FORMAT: "hdc"}


def _dev_check(A: _Matrix) -> None:
    if A.device.type != "cuda":
        raise NotImplementedException("convert: containers must live on a CUDA device")


def _call(name, *args):
    _lib.call(name, *args)


def _empty(n, dtype, device) -> torch.Tensor:
    return torch.empty(int(n), dtype=dtype, device=device)


def _arrays(A: _Matrix):
    for v in vars(A).values():
        if isinstance(v, torch.Tensor):
            yield v
        elif isinstance(v, _Matrix):
            yield from _arrays(v)


def _run(stream, work, src: _Matrix, *args):
    """work(src, *args) on `stream`: everything it allocates comes from that
    stream's own memory (a block that torch has just freed may still be in use
    on the stream that it belongs to, and on no other), src's arrays are kept
    until the stream has read them, and the result's until the caller's stream,
    where it is used next, is done with them."""
    if stream is None or src.device.type != "cuda":
        return work(src, *args)
    if not isinstance(stream, torch.cuda.Stream):
        handle = int(stream)
        stream = torch.cuda.ExternalStream(handle) if handle else torch.cuda.default_stream()
    caller, read = torch.cuda.current_stream(), list(_arrays(src))
    if caller.cuda_stream == stream.cuda_stream:
        return work(src, *args)
    with torch.cuda.stream(stream):
        try:
            out = work(src, *args)
        finally:
            for t in read:
                if t.is_cuda:
                    t.record_stream(stream)
    for t in _arrays(out if isinstance(out, _Matrix) else src):  # src: changed in place
        if t.is_cuda:
            t.record_stream(caller)
    return out


def to_coo(A: _Matrix, stream=None) -> CooMatrix:
    """Any container -> a new COO container (the reference's X -> COO)."""
    return _run(stream, _to_coo, A)


def _to_coo(A: _Matrix) -> CooMatrix:
    if isinstance(A, DynamicMatrix):
        A = A.active()
    _dev_check(A)
    _suffix(A.dtype)
    if A.FORMAT == COO_FORMAT:
        return CooMatrix(A.nrows(), A.ncols(), A.nnnz(), A.row_indices().clone(), A.column_indices().clone(),
                         A.values().clone(), A.dtype, A.device)
    z = A.nnnz()  # the conversions write every entry: nothing to clear
    return _fill_coo(A, _empty(z, torch.int32, A.device), _empty(z, A.dtype, A.device))


def _fill_coo(A: _Matrix, cols: torch.Tensor, vals: torch.Tensor) -> CooMatrix:
    out = CooMatrix(A.nrows(), A.ncols(), A.nnnz(), _empty(A.nnnz(), torch.int32, A.device), cols, vals, A.dtype,
                    A.device)
    sd, dd = A._desc(), out._desc()
    _call(f"mgb_convert_{_NAME[A.FORMAT]}_to_coo_{_suffix(A.dtype)}", C.byref(sd), C.byref(dd),
          _stream_handle(None))
    return out


# Containers that a conversion fills: it writes every index, offset and value
# (padding included), so their arrays are not cleared first.

def _new_csr(n, m, z, dt, dev) -> CsrMatrix:
    return CsrMatrix(n, m, z, _empty(n + 1, torch.int32, dev), _empty(z, torch.int32, dev), _empty(z, dt, dev), dt, dev)


def _new_coo(n, m, z, dt, dev) -> CooMatrix:
    return CooMatrix(n, m, z, _empty(z, torch.int32, dev), _empty(z, torch.int32, dev), _empty(z, dt, dev), dt, dev)


def _new_dia(n, m, z, nd, dt, dev) -> DiaMatrix:
    return DiaMatrix(n, m, z, nd, diagonal_offsets=_empty(nd, torch.int32, dev),
                     values=_empty(get_pad_size(n, 32) * nd, dt, dev), dtype=dt, device=dev)


def _new_ell(n, m, z, w, dt, dev) -> EllMatrix:
    slab = n * get_pad_size(w, 32)
    return EllMatrix(n, m, z, w, column_indices=_empty(slab, torch.int32, dev), values=_empty(slab, dt, dev), dtype=dt,
                     device=dev)


def from_coo(coo: CooMatrix, fmt: int, hyb_width: int = 0, stream=None) -> _Matrix:
    """COO -> a new container of format `fmt` (the reference's COO -> Y)."""
    return _run(stream, _from_coo, coo, fmt, hyb_width)


def _from_coo(coo: CooMatrix, fmt: int, hyb_width: int) -> _Matrix:
    _dev_check(coo)
    sfx = _suffix(coo.dtype)
    sh = _stream_handle(None)
    sd = coo._desc()
    n, m, z, dt, dev = coo.nrows(), coo.ncols(), coo.nnnz(), coo.dtype, coo.device
    fmt = int(fmt)
    if fmt == COO_FORMAT:
        return _to_coo(coo)
    if fmt not in _NAME:
        raise NotImplementedException(f"format {fmt}")
    nb, plan = C.c_int64(), _lib.CooPlan()
    _call("mgb_convert_coo_workspace_bytes", C.byref(sd), fmt, C.byref(nb))
    ws = _empty(nb.value, torch.uint8, dev)
    # sizes known before the plan: allocate while the GPU still has work queued
    out = _new_csr(n, m, z, dt, dev) if fmt == CSR_FORMAT else None
    _call("mgb_convert_coo_plan", C.byref(sd), fmt, int(hyb_width), _ptr(ws), nb.value, C.byref(plan), sh)
    out = out or _planned_container(coo, fmt, plan)
    dd = out._desc()
    fill = _empty(plan.fill_bytes, torch.uint8, dev) if plan.fill_bytes else None
    _call(f"mgb_convert_coo_planned_{sfx}", C.byref(sd), C.byref(plan), C.byref(dd), _ptr(fill), plan.fill_bytes, sh)
    return out


def _planned_container(src: _Matrix, fmt: int, plan) -> _Matrix:
    n, m, z, dt, dev = src.nrows(), src.ncols(), src.nnnz(), src.dtype, src.device
    s0, s1, s2 = plan.sizes
    if fmt == DIA_FORMAT:
        return _new_dia(n, m, z, s0, dt, dev)
    if fmt == ELL_FORMAT:
        return _new_ell(n, m, z, s0, dt, dev)
    if fmt == HYB_FORMAT:
        return HybMatrix(_new_ell(n, m, s1, s0, dt, dev), _new_coo(n, m, s2, dt, dev), dt, dev)
    return HdcMatrix(_new_dia(n, m, s1, s0, dt, dev), _new_csr(n, m, s2, dt, dev), dt, dev)


def _from_csr(A: CsrMatrix, fmt: int, hyb_width: int) -> _Matrix:
    """CSR -> a new DIA / ELL / HYB / HDC container, as through COO but without
    its row indices (which are made where the library has no such path)."""
    _dev_check(A)
    sfx, sh, sd = _suffix(A.dtype), _stream_handle(None), A._desc()
    if fmt in (DIA_FORMAT, ELL_FORMAT, HYB_FORMAT, HDC_FORMAT):
        nb, plan = C.c_int64(), _lib.CooPlan()
        _call("mgb_convert_csr_workspace_bytes", C.byref(sd), fmt, C.byref(nb))
        ws = _empty(nb.value, torch.uint8, A.device)
        _call(f"mgb_convert_csr_plan_{sfx}", C.byref(sd), fmt, int(hyb_width), _ptr(ws), nb.value, C.byref(plan), sh)
        if plan.format:
            out = _planned_container(A, fmt, plan)
            dd = out._desc()
            _call(f"mgb_convert_csr_planned_{sfx}", C.byref(sd), C.byref(plan), C.byref(dd), sh)
            return out
    return _from_coo(_fill_coo(A, A.column_indices(), A.values()), fmt, hyb_width)


def _convert_to(A: _Matrix, fmt: int, hyb_width: int) -> _Matrix:
    """A in another format, through COO as the reference does."""
    if fmt == COO_FORMAT:
        return _to_coo(A)
    if A.FORMAT == CSR_FORMAT:
        return _from_csr(A, fmt, hyb_width)
    return _from_coo(A if A.FORMAT == COO_FORMAT else _to_coo(A), fmt, hyb_width)


def convert(src, dst, stream=None, hyb_width: int = 0):
    """convert(src, dst) fills container dst; convert(dyn, fmt) converts in place."""
    if isinstance(dst, (int, formats_e)) and not isinstance(dst, bool):
        return convert_inplace(src, dst, stream=stream, hyb_width=hyb_width)
    if isinstance(src, DynamicMatrix):
        src = src.active()
    target = dst.active_index() if isinstance(dst, DynamicMatrix) else dst.FORMAT
    if src.FORMAT == target:
        out = to_coo(src, stream) if target == COO_FORMAT else _deep_copy(src)
    else:
        out = _run(stream, _convert_to, src, target, hyb_width)
    if isinstance(dst, DynamicMatrix):
        dst.assign(out)
    else:
        dst.__dict__.update(out.__dict__)
    return dst


def _deep_copy(A: _Matrix) -> _Matrix:
    from .containers import matrix_from_host, matrix_to_host
    return matrix_from_host(matrix_to_host(A), device=A.device, dtype=A.dtype)


def convert_inplace(dyn: DynamicMatrix, fmt, stream=None, hyb_width: int = 0) -> conversion_error_e:
    """core/src/Morpheus_Convert.hpp:88-124.  fmt = AUTO_FORMAT (-1) asks the
    learned selector for the target format."""
    fmt = int(fmt)
    if fmt == -1:
        from .selector import select_format
        fmt = select_format(dyn)
    if fmt < 0 or fmt >= NFORMATS:
        return conversion_error_e.PROXY_TO_DYNAMIC
    if dyn.active_index() == fmt:
        return conversion_error_e.CONV_SUCCESS
    return _run(stream, _convert_inplace, dyn, fmt, hyb_width)


def _convert_inplace(dyn: DynamicMatrix, fmt: int, hyb_width: int) -> conversion_error_e:
    src = dyn.active()
    try:
        _dev_check(src)
        _suffix(src.dtype)
        if fmt == COO_FORMAT or src.FORMAT not in (COO_FORMAT, CSR_FORMAT):
            src = _to_coo(src)
    except MorpheusException:
        return conversion_error_e.DYNAMIC_TO_PROXY
    try:
        out = src if fmt == COO_FORMAT else _convert_to(src, fmt, hyb_width)
    except MorpheusException:
        return conversion_error_e.PROXY_TO_DYNAMIC
    dyn.assign(out)
    return conversion_error_e.CONV_SUCCESS


def sort_by_row_and_column(A: CooMatrix, stream=None) -> None:
    _run(stream, _sort, A)


def _sort(A: CooMatrix) -> None:
    _dev_check(A)
    d, nb = A._desc(), C.c_int64()
    _call("mgb_coo_sort_workspace_bytes", C.byref(d), C.byref(nb))
    ws = _empty(nb.value, torch.uint8, A.device)
    _call(f"mgb_coo_sort_by_row_and_column_ws_{_suffix(A.dtype)}", C.byref(d), _ptr(ws), nb.value,
          _stream_handle(None))


def is_sorted(A: CooMatrix, stream=None) -> bool:
    _dev_check(A)
    d = A._desc()
    out = C.c_int()
    _call("mgb_coo_is_sorted", C.byref(d), C.byref(out), _stream_handle(stream))
    return bool(out.value)


__all__ = ["convert", "convert_inplace", "to_coo", "from_coo", "sort_by_row_and_column", "is_sorted"]
