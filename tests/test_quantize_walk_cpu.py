"""How the streaming quantizer goes through large inputs (no GPU needed to ask)."""
from __future__ import annotations

import ctypes

import pytest

from test_abi_cpu import lib_path  # noqa: F401  (a fixture)

FP32, FP16, BF16 = 0, 1, 2
MARK, BACKWARD = 1, 2


@pytest.fixture(scope="module")
def walk(lib_path):  # noqa: F811
    fn = ctypes.CDLL(lib_path).ck_debug_quantize_nvfp4_walk
    fn.argtypes, fn.restype = [ctypes.c_int, ctypes.c_int, ctypes.c_int64, ctypes.c_int64], ctypes.c_int
    return fn


@pytest.mark.parametrize("dtype, rows, cols, dynamic, static", [
    (FP32, 2730, 3072, 0, 0), (FP32, 2731, 3072, MARK, MARK),                          # 32 MiB of input
    (FP32, 10240, 3072, MARK, MARK), (FP32, 10241, 3072, MARK | BACKWARD, MARK),       # 120 MiB of input
    (FP32, 38836, 3072, MARK | BACKWARD, MARK), (FP32, 38837, 3072, 0, 0),             # 64 MiB of codes and scales
    (FP32, 130, 262144, MARK | BACKWARD, MARK),
    (BF16, 5461, 3072, 0, 0), (BF16, 5462, 3072, MARK, MARK), (FP16, 36864, 3072, MARK, MARK), (BF16, 38837, 3072, 0, 0),
])
def test_lines(walk, dtype, rows, cols, dynamic, static):
    assert walk(dtype, 1, rows, cols) == dynamic and walk(dtype, 0, rows, cols) == static
