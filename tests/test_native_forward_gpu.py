"""Layers whose forward goes through the native half of the CUDA wrappers, held against the layout path."""
from __future__ import annotations

import pytest
import torch
import torch.nn as nn
from torch.nn.utils import parametrize

pytestmark = pytest.mark.gpu


def _layer(layout, k, n, bias, device):
    from comfy_kitchen.modules import MXFP8Linear, NVFP4Linear

    gen = torch.Generator(device=device).manual_seed(k + n)
    dense = nn.Linear(k, n, bias=bias, device=device, dtype=torch.bfloat16)
    with torch.no_grad():
        dense.weight.copy_(torch.randn(n, k, generator=gen, device=device) * 0.02)
        if bias:
            dense.bias.copy_(torch.linspace(-1, 1, n, device=device))
    return (NVFP4Linear if layout == "nvfp4" else MXFP8Linear).from_linear(dense)


def _x(m, k, device):
    gen = torch.Generator(device=device).manual_seed(m)
    return torch.randn(m, k, generator=gen, device=device).bfloat16()


class _Doubled(nn.Module):
    def forward(self, bias):
        return 2 * bias


@pytest.mark.parametrize("held", ["buffer", "parametrized"])
@pytest.mark.parametrize("m", [3, 200])
@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_bias_wherever_the_layer_holds_it(cuda_device, layout, m, held):
    layer, x = _layer(layout, 256, 128, True, cuda_device), _x(m, 256, cuda_device)
    bias = layer.bias.detach()
    with torch.inference_mode():
        plain = layer(x)
    if held == "buffer":
        del layer.bias
        layer.register_buffer("bias", bias)
    else:
        parametrize.register_parametrization(layer, "bias", _Doubled())
        layer.parametrizations.bias.original.data.div_(2)  # a power of two: the same bias
    with torch.inference_mode():
        assert torch.equal(layer(x), plain)


@pytest.mark.parametrize("m, n", [(1, 1000), (8, 200), (40, 1000), (300, 1000)])
@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_padded_out_features(cuda_device, monkeypatch, layout, m, n):
    """out_features that are no whole blocks, without a bias: the layout path's bits from one native call."""
    from comfy_kitchen.backends import cuda as backend
    from comfy_kitchen.modules import _QuantizedLinearBase

    layer, x = _layer(layout, 512, n, False, cuda_device), _x(m, 512, cuda_device)
    name = f"linear_{layout}_from_float"
    native, taken = backend._host, []

    class Counting:
        def __getattr__(self, attribute):
            fn = getattr(native, attribute)
            if attribute != name:
                return fn

            def call(*args):
                out = fn(*args)
                taken.append(out is not None)
                return out
            return call

    with torch.inference_mode():
        want = _QuantizedLinearBase.forward(layer, x)
        monkeypatch.setattr(backend, "_host", Counting())
        got = layer(x)
    assert got.shape == (m, n) and torch.equal(got, want)
    assert taken == [True]
