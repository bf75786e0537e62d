"""The C-ABI library loads on a machine without a GPU and exports exactly what
include/b200ops.h declares (no compute calls here)."""

import ctypes
import os
import re

from backendbench_b200 import _abi
from conftest import ROOT


def _declared():
    text = open(os.path.join(ROOT, "include", "b200ops.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(b200_[a-z0-9_]+)\s*\(", text)))


def test_library_loads_and_reports_version():
    lib = _abi.lib()
    assert lib.b200_abi_version() == _abi.ABI_VERSION == 1
    assert lib.b200_strerror(0) == b"ok"
    assert b"dtype" in lib.b200_strerror(-2)


def test_every_declared_symbol_is_exported_and_bound():
    names = _declared()
    assert len(names) >= 23
    handle = ctypes.CDLL(_abi.LIB_PATH)
    for n in names:
        assert hasattr(handle, n), f"{n} declared in include/b200ops.h but not exported"
    assert set(names) == set(_abi.SIGNATURES), set(names) ^ set(_abi.SIGNATURES)


def test_argument_validation_needs_no_gpu():
    lib = _abi.lib()
    shape = _abi.i64_array([4])
    # unsupported dtype and bad rank are rejected before anything touches the device
    assert lib.b200_relu(None, None, 1, shape, shape, _abi.I64, None) == -2
    assert lib.b200_relu(None, None, 99, shape, shape, _abi.F32, None) == -1
    assert lib.b200_softmax(None, None, -1, 4, 1, _abi.F32, _abi.F32, 0, None) == -1
    assert lib.b200_reduce_scratch_bytes(1, 1 << 26, 1) > 0
    assert lib.b200_reduce_scratch_bytes(8192, 4096, 1) == 0
    assert lib.b200_gemm(None, None, None, None, 1, 0, 5, 5, 0, 5, 1, 0, 5, 1, 0, 0, 1.0, 0.0, _abi.F32, None, None) == 0


def test_nothing_to_compare_is_close_whatever_its_dtype():
    lib = _abi.lib()
    rec = ctypes.c_int64(0)  # (not written: the record is not to be reset)
    for dtype in (_abi.F32, _abi.I64, _abi.F64, 99):
        assert lib.b200_allclose(None, None, 0, dtype, 0.0, 0.0, ctypes.addressof(rec), 0, None) == 0
    assert lib.b200_allclose(ctypes.addressof(rec), ctypes.addressof(rec), 1, 99, 0.0, 0.0, ctypes.addressof(rec), 0, None) == -2


STRIP, WIDE, ROWS, BINS, BUCKETS, CHAINS, LINES = range(1, 8)


def _scatter_path(shape, ishape, dim, dtype, base=1 << 20, columns=False):
    """Which kernels serve a scatter_add, and what scratch it asks for, of tensors at (aligned) addresses that nobody looks behind.
    `columns`: index and src are laid out along their second-to-last dim."""
    strides = [1]
    for n in reversed(ishape[1:]):
        strides.insert(0, strides[0] * n)
    if columns:
        strides[-2:] = [1, ishape[-2]]
    a = [_abi.i64_array(v) for v in (shape, ishape, strides, strides)]
    args = (base, base, base, base, len(shape), *a, dim, dtype)
    return _abi.lib().b200_scatter_add_path(*args), _abi.lib().b200_scatter_add_scratch_bytes(*args)


def test_strips_go_on_where_bins_do_not_pay():
    """65 to 127 rows of many columns on the strips' grid: bins would be the faster ones, were they open to them."""
    for shape in ([100, 8192], [65, 40000], [127, 16384], [2, 100, 8192]):
        assert _scatter_path(shape, shape, len(shape) - 2, _abi.F32) == (STRIP, 0), shape
    assert _scatter_path([4000, 512], [4000, 512], 0, _abi.F32)[0] == _scatter_path([2000, 256], [2000, 256], 0, _abi.F32)[0] == BINS
    for shape, rows in (([969, 252], 969), ([1951, 140], 975), ([500, 512], 500)):
        assert _scatter_path(shape, [rows, shape[1]], 0, _abi.F16) == (STRIP, 0), shape
    assert _scatter_path([4096, 4096], [4096, 4096], 0, _abi.F32) == (WIDE, 0)


def test_short_lines_side_by_side_stay_lines():
    """25 to 64 source rows go through bins where there are few columns to walk them, however many dims these are dealt out over."""
    path = lambda s: _scatter_path(s, s, len(s) - 2, _abi.F32)[0]
    assert path([60, 333]) == path([4, 60, 333]) == path([1, 60, 2047]) == BINS
    assert path([24, 333]) == path([60, 2049]) == path([267, 64, 23]) == path([145, 42, 565]) == LINES


def test_which_matrices_go_through_bins():
    """The shapes of the bit-exact tests on a GPU, and those on either side of the rules."""
    for dtype in (_abi.F32, _abi.BF16, _abi.F16):
        for shape, ishape, dim in (((5003, 33), (5003, 33), 0), ((129, 31), (700, 31), 0), ((20001, 40), (20001, 40), 0), ((600, 65), (20000, 65), 0), ((5, 701, 37), (4, 650, 35), 1),
                                   ((4100, 70), (2050, 70), 0), ((4100, 45), (4100, 45), 0), ((40, 2), (3001, 2), 0), ((150134, 63), (75067, 63), 0)):
            assert _scatter_path(shape, ishape, dim, dtype)[0] == BINS, shape
        assert _scatter_path((4100, 45), (4100, 45), 0, dtype, columns=True)[0] == BINS
        assert _scatter_path((300, 2), (3001, 2), 0, dtype)[0] == BUCKETS  # more bins than there is room to count in
        assert _scatter_path((200000, 63), (100000, 63), 0, dtype)[0] == CHAINS
        assert _scatter_path((70001,), (70001,), 0, dtype)[0] in (ROWS, CHAINS)
