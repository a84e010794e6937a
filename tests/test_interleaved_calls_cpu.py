"""Calls of several launches from two threads that share a stream: what passes from one launch to the next is
in memory of that call alone.  The library is replaced by one that computes on the host and lets every call
make its first launch before any makes its second, which is the order that threads can produce."""
from __future__ import annotations

import contextlib
import ctypes
import threading

import numpy as np
import pytest
import torch


class Interleaved:
    """First launch: the input's largest magnitude to the scratch; second: from there to the result."""

    def __init__(self, threads: int):
        self.barrier = threading.Barrier(threads)

    @staticmethod
    def _read(p, n=1):
        return np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_float)), (n,))

    def _two_launches(self, x, n, scratch, out):
        self._read(scratch)[0] = np.abs(self._read(x, n)).max()
        self.barrier.wait(timeout=20)
        self._read(out)[0] = self._read(scratch)[0]
        return 0

    def ck_quantize_nvfp4_dynamic_scratch_bytes(self, n):
        return 4096

    def ck_linear_nvfp4_from_float_workspace_bytes(self, m, k, dynamic):
        return 4096

    def ck_linear_mxfp8_from_float_workspace_bytes(self, m, k):
        return 4096

    def ck_quantize_nvfp4_dynamic(self, x, dtype, scale, codes, scales, rows, cols, out_rows, out_cols, hi, scratch, nbytes, stream):
        return self._two_launches(x, rows * cols, scratch, scale)

    def ck_linear_nvfp4_from_float(self, x, dtype, sx, w, sw, tsw, bias, bias_dtype, out, out_dtype, m, n, k, ws, nbytes, stream):
        return self._two_launches(x, m * k, ws, out)

    def ck_linear_mxfp8_from_float(self, x, dtype, w, sw, bias, bias_dtype, out, out_dtype, m, n, k, ws, nbytes, stream):
        return self._two_launches(x, m * k, ws, out)


def _call(backend, entry, x):
    n, k = 128, x.shape[1]
    scale = torch.ones(())
    if entry == "quantize_nvfp4_dynamic":
        return backend.quantize_nvfp4_dynamic(x)[2]
    if entry == "linear_nvfp4_from_float":
        scales = torch.zeros(n, k // 16, dtype=torch.uint8)
        return backend.linear_nvfp4_from_float(x, torch.zeros(n, k // 2, dtype=torch.uint8), scale, scales, out_dtype=torch.float32)
    scales = torch.zeros(n, k // 32, dtype=torch.uint8)
    return backend.linear_mxfp8_from_float(x, torch.zeros(n, k, dtype=torch.uint8), scales, out_dtype=torch.float32)


@pytest.mark.parametrize("entry", ["quantize_nvfp4_dynamic", "linear_nvfp4_from_float", "linear_mxfp8_from_float"])
def test_threads_of_one_stream_keep_their_own_intermediates(entry, monkeypatch):
    from comfy_kitchen.backends import cuda as backend

    lib = Interleaved(threads=1)
    monkeypatch.setattr(backend, "_lib", lib)
    monkeypatch.setattr(backend, "load_library", lambda: lib)
    monkeypatch.setattr(backend, "_stream", lambda device: 0)
    monkeypatch.setattr(backend, "_capturing", lambda: False)
    monkeypatch.setattr(backend, "_on_device", lambda device: contextlib.nullcontext())
    backend._workspace_bytes.cache_clear()
    _call(backend, entry, torch.ones(128, 256))  # buffers that are kept from call to call exist now
    lib.barrier = threading.Barrier(2)
    got = {}

    def work(value):
        got[value] = float(_call(backend, entry, torch.full((128, 256), value)).flatten()[0])  # 128 KiB

    threads = [threading.Thread(target=work, args=(v,)) for v in (1.0, 1000.0)]
    try:
        for t in threads:
            t.start()
    finally:
        for t in threads:
            t.join(timeout=30)
        backend._workspace_bytes.cache_clear()
    assert got == {1.0: 1.0, 1000.0: 1000.0}
