"""What the layers hand to the native half of the CUDA wrappers (a stand-in for it here: the values are not looked at)."""
from __future__ import annotations

import pytest
import torch
import torch.nn as nn
from torch.nn.utils import parametrize

from comfy_kitchen import modules
from comfy_kitchen.tensor import QuantizedTensor, TensorCoreMXFP8Layout, TensorCoreNVFP4Layout


class _Host:
    """Takes every call: a result of the weight's physical rows."""

    def __init__(self):
        self.calls = []

    def linear_nvfp4_from_float(self, x, w, w_scale, w_block_scales, bias, x_scale, out_dtype):
        return self._take(x, w, bias, out_dtype)

    def linear_mxfp8_from_float(self, x, w, w_block_scales, bias, out_dtype):
        return self._take(x, w, bias, out_dtype)

    def _take(self, x, w, bias, out_dtype):
        self.calls.append(bias)
        return torch.arange(float(w.shape[0])).to(out_dtype).expand(x.shape[0], w.shape[0]).contiguous()


def _layer(layout, out_features=32, in_features=64, bias=True):
    if layout == "nvfp4":
        layer, rows = modules.NVFP4Linear(in_features, out_features, bias=bias), (out_features + 15) // 16 * 16
        params = TensorCoreNVFP4Layout.Params(scale=torch.ones(()), orig_dtype=torch.bfloat16, orig_shape=(out_features, in_features),
                                              block_scale=torch.ones(128, 4).to(torch.float8_e4m3fn))
        w = QuantizedTensor(torch.zeros(rows, in_features // 2, dtype=torch.uint8), "TensorCoreNVFP4Layout", params)
    else:
        layer, rows = modules.MXFP8Linear(in_features, out_features, bias=bias), (out_features + 31) // 32 * 32
        params = TensorCoreMXFP8Layout.Params(scale=torch.full((128, 4), 127, dtype=torch.uint8).view(torch.float8_e8m0fnu),
                                              orig_dtype=torch.bfloat16, orig_shape=(out_features, in_features))
        w = QuantizedTensor(torch.zeros(rows, in_features).to(torch.float8_e4m3fn), "TensorCoreMXFP8Layout", params)
    layer.weight = nn.Parameter(w, requires_grad=False)
    if bias:
        layer.bias = nn.Parameter(torch.arange(float(out_features)), requires_grad=False)
    return layer


@pytest.fixture
def host(monkeypatch):
    host = _Host()
    monkeypatch.setattr(modules, "host_half", lambda: host)
    return host


class _Doubled(nn.Module):
    def forward(self, bias):
        return 2 * bias


@pytest.mark.parametrize("held", ["parameter", "buffer", "parametrized", "none"])
@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_bias_wherever_the_layer_holds_it(host, layout, held):
    layer = _layer(layout, bias=held != "none")
    if held == "buffer":
        b = layer.bias.detach()
        del layer.bias
        layer.register_buffer("bias", b)
    elif held == "parametrized":
        parametrize.register_parametrization(layer, "bias", _Doubled())
    layer(torch.zeros(4, 64, dtype=torch.bfloat16))
    (got,) = host.calls
    assert got is None if held == "none" else torch.equal(got, layer.bias)


@pytest.mark.parametrize("out_features", [32, 40])  # 40: the weight has 48 or 64 rows
@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_padded_weight_rows_are_cut_from_the_native_result(host, layout, out_features):
    """One native call, whose result is the layer's."""
    y = _layer(layout, out_features, bias=False)(torch.zeros(4, 64, dtype=torch.bfloat16))
    assert len(host.calls) == 1
    assert y.shape == (4, out_features) and torch.equal(y[3], torch.arange(float(out_features)).bfloat16())


@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_layers_ask_the_backend_s_own_half(monkeypatch, layout):
    """Without the stand-in for the function that finds it."""
    from comfy_kitchen.backends import cuda as backend

    host = _Host()
    monkeypatch.setattr(backend, "_host", host)
    layer = _layer(layout)
    assert torch.equal(layer(torch.zeros(3, 64)), torch.arange(32.0).expand(3, 32)) and len(host.calls) == 1
