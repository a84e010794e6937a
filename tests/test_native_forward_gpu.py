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


@pytest.mark.parametrize("shape", [(2, 3, 512), (1, 40, 512), (3, 100, 512), (2, 1, 2, 4, 512), (1, 1, 512)])
@pytest.mark.parametrize("n", [256, 200])
@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_activations_of_any_rank(cuda_device, layout, n, shape):
    """The rows' bits in the activation's shape, strides as the 2-D result has them, natively and through the Python route."""
    from comfy_kitchen.backends import cuda as backend
    from comfy_kitchen.modules import _QuantizedLinearBase

    layer, flat = _layer(layout, 512, n, n == 256, cuda_device), _x(torch.Size(shape).numel() // 512, 512, cuda_device)
    x = flat.view(shape)
    with torch.inference_mode():
        want = layer(flat)
        got = layer(x)
        assert got.shape == (*shape[:-1], n) and torch.equal(got.reshape(-1, n), want)
        strides = [t.stride()[i] for t in (got, want.view(got.shape)) for i in range(len(shape)) if shape[i] > 1]
        assert strides[: len(strides) // 2] == strides[len(strides) // 2 :]
        assert torch.equal(got, _QuantizedLinearBase.forward(layer, x))
        apart = torch.stack([x, x], dim=-1)[..., 0]  # not contiguous: the Python route
        assert not apart.is_contiguous() and torch.equal(layer(apart), got)
    w = layer.weight
    args = (w._params.scale, w._params.block_scale) if layout == "nvfp4" else (w._params.scale,)
    with pytest.raises(AssertionError):  # the wrapper itself takes a matrix
        getattr(backend, f"linear_{layout}_from_float")(x, w._qdata, *args)


@pytest.mark.parametrize("layout", ["nvfp4", "mxfp8"])
def test_native_for_tokens_in_batches(cuda_device, layout):
    from comfy_kitchen.backends import cuda as backend

    layer, x = _layer(layout, 512, 256, True, cuda_device), _x(6, 512, cuda_device)
    w, bias = layer.weight, layer.bias
    native = getattr(backend._host, f"linear_{layout}_from_float")
    args = (w._params.scale, w._params.block_scale, bias, None, x.dtype) if layout == "nvfp4" else (w._params.scale, bias, x.dtype)
    assert native(x.view(2, 3, 512), w._qdata, *args).shape == (2, 3, 256)
    assert native(x[0], w._qdata, *args) is None and native(x.view(2, 3, 512)[:0], w._qdata, *args) is None
