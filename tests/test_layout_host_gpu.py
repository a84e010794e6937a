"""The layouts' route through the native half: the codes, the parameters and the results of the Python wrappers', and neither half where a
function of the backend has been replaced."""
from __future__ import annotations

import dataclasses

import pytest
import torch

from comfy_kitchen.tensor import QuantizedTensor

pytestmark = pytest.mark.gpu

LAYOUTS = ["TensorCoreNVFP4Layout", "TensorCoreMXFP8Layout"]


@pytest.fixture
def backend(cuda_device):
    from comfy_kitchen.backends import cuda as backend

    assert backend._host is not None, "lib/_ck_host.so is not built or does not load"
    return backend


def _same(a, b):
    assert type(a) is type(b)
    if not isinstance(a, torch.Tensor):
        assert a == b
        return
    assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride() and a.device == b.device and a.requires_grad == b.requires_grad
    assert torch.equal(a.view(torch.uint8) if a.dim() else a, b.view(torch.uint8) if b.dim() else b)


def _same_quantized(a, b):
    if isinstance(a, str):
        assert a == b
        return
    _same(a._qdata, b._qdata)
    for field in dataclasses.fields(a._params):
        _same(getattr(a._params, field.name), getattr(b._params, field.name))


# one row, both sides of 64 KiB and of 128 KiB in 16-bit types (fp32: twice that), ragged rows, ragged columns, more than a tile
SHAPES = [(1, 64), (8, 4096), (8, 4128), (16, 4096), (16, 4128), (33, 70), (77, 256), (300, 96)]


@pytest.mark.parametrize("inference", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows, cols", SHAPES)
def test_same_as_the_python_wrappers(backend, cuda_device, monkeypatch, rows, cols, dtype, inference):
    gen = torch.Generator(device=cuda_device).manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device).to(dtype)
    w, padded_w = (torch.randn(n, cols, generator=gen, device=cuda_device).to(dtype) for n in (256, 200))
    given = torch.tensor(0.02, device=cuda_device)
    scales = [None, given, torch.nn.Parameter(given.clone(), requires_grad=False), given.half(), given.reshape(1), given.cpu(), 0.02, "recalculate"]
    inputs = [x, torch.nn.Parameter(x.clone(), requires_grad=False), x.t().contiguous().t()]  # the last one is refused unless it has one row

    def from_float(*args, **kwargs):
        try:
            return QuantizedTensor.from_float(*args, **kwargs)
        except AssertionError as e:
            return str(e)

    def calls():
        quantized = [from_float(t, LAYOUTS[0], scale=s) for t in inputs for s in scales]
        quantized += [from_float(t, LAYOUTS[1]) for t in inputs]
        results = []
        for layout in LAYOUTS:
            qx, qw, padded_qw = (QuantizedTensor.from_float(t, layout) for t in (x, w, padded_w))
            results += [torch.nn.functional.linear(qx, qw, torch.linspace(-1, 1, 256, device=cuda_device).to(dtype)), torch.nn.functional.linear(qx, padded_qw)]
        return quantized, results

    with torch.inference_mode(inference):
        got, got_results = calls()
        monkeypatch.setattr(backend, "_host", None)
        want, want_results = calls()
        for a, b in zip(got, want):
            _same_quantized(a, b)
        for a, b in zip(got_results, want_results):
            _same(a, b)
    assert got[1]._params.scale is given and got[2]._params.scale is scales[2]


@pytest.mark.parametrize("name", ["quantize_nvfp4", "quantize_nvfp4_dynamic", "quantize_mxfp8", "scaled_mm_nvfp4", "scaled_mm_mxfp8"])
def test_a_replaced_function_is_called(backend, cuda_device, monkeypatch, name):
    x, w = (torch.randn(r, 256, device=cuda_device, dtype=torch.bfloat16) for r in (300, 128))  # more than 128 KiB
    layout = LAYOUTS["mxfp8" in name]
    weight = QuantizedTensor.from_float(w, layout)
    calls, stock = [], getattr(backend, name)

    def replacement(*args, **kwargs):
        calls.append(name)
        return stock(*args, **kwargs)

    def call():
        kwargs = {"scale": torch.tensor(0.02, device=cuda_device)} if name == "quantize_nvfp4" else {}
        with torch.inference_mode():
            return torch.nn.functional.linear(QuantizedTensor.from_float(x, layout, **kwargs), weight)

    want = call()
    monkeypatch.setattr(backend, name, replacement)
    assert torch.equal(call(), want) and calls == [name]
    monkeypatch.undo()
    assert torch.equal(call(), want) and calls == [name]
