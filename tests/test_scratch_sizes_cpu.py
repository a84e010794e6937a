"""Size queries of the C ABI (no GPU needed)."""
from __future__ import annotations

import ctypes

import pytest

from test_abi_cpu import lib_path  # noqa: F401  (a fixture)


@pytest.fixture(scope="module")
def lib(lib_path):  # noqa: F811
    lib = ctypes.CDLL(lib_path)
    for name in ("ck_quantize_nvfp4_dynamic_scratch_bytes", "ck_nvfp4_tensor_scale_scratch_bytes"):
        getattr(lib, name).argtypes, getattr(lib, name).restype = [ctypes.c_int64], ctypes.c_int64
    lib.ck_linear_nvfp4_from_float_workspace_bytes.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int]
    lib.ck_linear_nvfp4_from_float_workspace_bytes.restype = ctypes.c_int64
    return lib


@pytest.mark.parametrize("n", [1, 16, 16384, 16385, 592 * 16384, 592 * 16384 + 1, 4096 * 3072, 16384 * 8192, 1 << 30, 1 << 33])
def test_dynamic_scratch_depends_on_the_input_alone(lib, n):
    """One fp32 partial per 64 KiB of the input up to 592 of them, per 32 KiB beyond, at most 16384, behind a
    256-byte head (or what the one-kernel scale wants): no term in the SM count of whichever device happens
    to be current.  The input may be fp32."""
    partials = -(-4 * n // 65536)
    if partials > 592:
        partials = min(-(-4 * n // 32768), 16384)
    assert lib.ck_quantize_nvfp4_dynamic_scratch_bytes(n) == max(256 + 4 * partials, lib.ck_nvfp4_tensor_scale_scratch_bytes(n))


@pytest.mark.parametrize("rows, kib", [(1, 64), (8, 64), (9, 128), (1 << 20, 128)])
def test_inputs_that_are_read_whole(lib, rows, kib):
    lib.ck_quantize_nvfp4_dynamic_whole_input_bytes.argtypes = [ctypes.c_int64]
    lib.ck_quantize_nvfp4_dynamic_whole_input_bytes.restype = ctypes.c_int64
    assert lib.ck_quantize_nvfp4_dynamic_whole_input_bytes(rows) == kib << 10


def test_one_row_has_the_lowest_line(lib):
    """Up to it the scratch is one that callers share: no number of rows may write to it."""
    lib.ck_quantize_nvfp4_dynamic_whole_input_bytes.restype = ctypes.c_int64
    line = lambda rows: lib.ck_quantize_nvfp4_dynamic_whole_input_bytes(ctypes.c_int64(rows))
    assert all(line(1) <= line(rows) for rows in (1, 2, 3, 7, 8, 9, 64, 1000, 32768))


def test_dynamic_scratch_of_nothing(lib):
    assert lib.ck_quantize_nvfp4_dynamic_scratch_bytes(0) == 0 == lib.ck_quantize_nvfp4_dynamic_scratch_bytes(-5)


@pytest.mark.parametrize("m, k, supported", [(1 << 15, 1 << 15, True), (1 << 20, 1 << 10, True), ((1 << 20) + 16, 1 << 10, False),
                                             (1 << 15, (1 << 15) + 32, False)])
def test_linear_takes_up_to_2_30_elements_with_a_dynamic_scale(lib, m, k, supported):
    """The limit that the header states, and a chunk of the reduction (16384 elements) or more above it."""
    assert (lib.ck_linear_nvfp4_from_float_workspace_bytes(m, k, 1) > 0) == supported
    assert lib.ck_linear_nvfp4_from_float_workspace_bytes(m, k, 0) > 0
    assert lib.ck_linear_nvfp4_from_float_workspace_bytes(m, k, 0) % 256 == 0


def test_one_mebibyte_does_all_but_huge_inputs(lib):
    """The wrappers' smallest buffer, handed in without asking for the size."""
    assert lib.ck_quantize_nvfp4_dynamic_scratch_bytes((1 << 31) - 1) <= 1 << 20
