"""Which library calls a dynamically scaled activation takes: one where the streaming quantizer applies, the
one-kernel scale on its zeroed scratch and the quantizer elsewhere (the one call would have to clear a counter
first, a launch more than before it existed)."""
from __future__ import annotations

import contextlib

import pytest
import torch


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        if name.endswith("_bytes"):
            return lambda *args: 4096
        return lambda *args: self.calls.append((name, args)) or 0


@pytest.fixture
def recorded(monkeypatch):
    from comfy_kitchen.backends import cuda as backend

    lib = Recorder()
    monkeypatch.setattr(backend, "_lib", lib)
    monkeypatch.setattr(backend, "load_library", lambda: lib)
    monkeypatch.setattr(backend, "_stream", lambda device: 0)
    monkeypatch.setattr(backend, "_capturing", lambda: False)
    monkeypatch.setattr(backend, "_on_device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(backend, "_scale_scratch", {})
    backend._workspace_bytes.cache_clear()
    yield backend, lib
    backend._workspace_bytes.cache_clear()


def _off_by_one(rows, cols, dtype):
    return torch.zeros(rows * cols + 1, dtype=dtype)[1:].view(rows, cols)


@pytest.mark.parametrize("x, pad, one_call", [
    (torch.zeros(16, 64, dtype=torch.bfloat16), False, True),
    (torch.zeros(5, 64, dtype=torch.bfloat16), True, True),        # rows padded, columns not
    (torch.zeros(16, 48), False, True),                            # fp32: whole 64-byte units
    (torch.zeros(16, 48, dtype=torch.float16), False, False),      # an odd number of blocks
    (torch.zeros(16, 65, dtype=torch.bfloat16), True, False),      # columns padded
    (torch.zeros(16, 65), True, False),
    (_off_by_one(16, 64, torch.bfloat16), False, False),           # not on 32 bytes
    (_off_by_one(16, 64, torch.float32), False, False),
])
def test_quantizer_route(recorded, x, pad, one_call):
    backend, lib = recorded
    codes, block_scales, scale = backend.quantize_nvfp4_dynamic(x, pad_16x=pad, hi_first=False)
    names = [name for name, _ in lib.calls]
    assert names == (["ck_quantize_nvfp4_dynamic"] if one_call else ["ck_nvfp4_tensor_scale", "ck_quantize_nvfp4"])
    rows, cols = (-(-d // 16) * 16 if pad else d for d in x.shape)
    assert codes.shape == (rows, cols // 2) and scale.shape == ()
    args = lib.calls[-1][1]
    assert args[5:9] == (*x.shape, rows, cols) and args[9] == 0 and args[2] in (scale.data_ptr(),)


@pytest.mark.parametrize("aligned", [True, False])
def test_linear_route(recorded, aligned):
    backend, lib = recorded
    x = torch.zeros(16, 64) if aligned else _off_by_one(16, 64, torch.float32)
    w, sw = torch.zeros(128, 32, dtype=torch.uint8), torch.zeros(128, 4, dtype=torch.uint8)
    backend.linear_nvfp4_from_float(x, w, torch.ones(()), sw)
    names = [name for name, _ in lib.calls]
    assert names == (["ck_linear_nvfp4_from_float"] if aligned else ["ck_nvfp4_tensor_scale", "ck_linear_nvfp4_from_float"])
    assert (lib.calls[-1][1][2] is None) == aligned
