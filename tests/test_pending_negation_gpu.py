"""Views whose negation is pending (the imaginary part of a conjugate) and symbolic zeros: their memory does not
hold their values, so they take the dispatcher's route, which materializes them."""
from __future__ import annotations

import pytest
import torch

import comfy_kitchen as ck

pytestmark = pytest.mark.gpu


def _negated(t: torch.Tensor) -> torch.Tensor:
    """-t as a strided view of complex memory."""
    view = torch.complex(torch.zeros_like(t), t).conj().imag
    assert view.is_neg() and torch.equal(view, -t)
    return view


def _same(got, want):
    for a, b in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
        assert torch.equal(a.view(torch.uint8) if a.element_size() == 1 else a, b.view(torch.uint8) if b.element_size() == 1 else b)


def test_pending_negation(cuda_device):
    gen = torch.Generator(device=cuda_device).manual_seed(1)
    x = torch.randn(48, 64, generator=gen, device=cuda_device)
    g = torch.tensor(0.01, device=cuda_device)
    bias = torch.linspace(-1, 1, 48, device=cuda_device)
    _same(ck.quantize_nvfp4(_negated(x), g), ck.quantize_nvfp4(-x, g))
    _same(ck.quantize_mxfp8(_negated(x)), ck.quantize_mxfp8(-x))
    codes, scales = ck.quantize_nvfp4(x, g)
    _same(ck.dequantize_nvfp4(codes, _negated(g), scales), ck.dequantize_nvfp4(codes, -g, scales))
    _same(ck.scaled_mm_nvfp4(codes, codes, g, _negated(g), scales, scales, bias=_negated(bias)),
          ck.scaled_mm_nvfp4(codes, codes, g, -g, scales, scales, bias=-bias))
    _same(ck.quantize_nvfp4(torch._neg_view(x), g), ck.quantize_nvfp4(-x, g))  # contiguous


def test_symbolic_zero(cuda_device):
    zero = torch._efficientzerotensor((16, 64), device=cuda_device, dtype=torch.float32)
    want = ck.quantize_mxfp8(torch.zeros(16, 64, device=cuda_device))
    _same(torch.ops.comfy_kitchen.quantize_mxfp8(torch.zeros(16, 64, device=cuda_device), False), want)
    try:
        through_dispatcher = torch.ops.comfy_kitchen.quantize_mxfp8(zero, False)
    except Exception as e:  # noqa: BLE001 - whatever the dispatcher makes of it, ck.* does the same
        with pytest.raises(type(e)):
            ck.quantize_mxfp8(zero)
    else:
        _same(ck.quantize_mxfp8(zero), through_dispatcher)
