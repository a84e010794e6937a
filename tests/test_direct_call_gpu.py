"""The operators of ``ck`` on plain CUDA tensors go straight to the registry: the same bits, types and errors
as through ``torch.ops``, and the dispatcher's route as soon as somebody watches or rewrites operator calls."""
from __future__ import annotations

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import comfy_kitchen as ck
from comfy_kitchen.exceptions import NoCapableBackendError
from comfy_kitchen.ops import DTYPE_TO_CODE, dispatcher_adds_nothing

pytestmark = pytest.mark.gpu


class Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


def _operands(device, m=40, n=128, k=256):
    gen = torch.Generator(device=device).manual_seed(3)
    x = torch.randn(m, k, generator=gen, device=device, dtype=torch.float32).bfloat16()
    w = torch.randn(n, k, generator=gen, device=device, dtype=torch.float32).bfloat16()
    return x, w, torch.tensor(0.01, device=device), torch.linspace(-1, 1, n, device=device)


def _same(a, b):
    assert type(a) is type(b) is torch.Tensor and a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride()
    assert a.requires_grad == b.requires_grad and not a._is_view() and not b._is_view()
    raw = (lambda t: t) if a.element_size() > 1 else (lambda t: t.view(torch.uint8))
    assert torch.equal(raw(a), raw(b))


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_same_as_through_the_dispatcher(cuda_device, fmt, out_dtype):
    x, w, g, bias = _operands(cuda_device)
    ops, code = torch.ops.comfy_kitchen, DTYPE_TO_CODE[out_dtype]
    if fmt == "nvfp4":
        qx, qw = ck.quantize_nvfp4(x, g, pad_16x=True), ck.quantize_nvfp4(w, g)
        pairs = list(zip(qx, ops.quantize_nvfp4(x, g, 0.0, True, True)))
        pairs.append((ck.scaled_mm_nvfp4(qx[0], qw[0], g, g, qx[1], qw[1], bias=bias, out_dtype=out_dtype),
                      ops.scaled_mm_nvfp4(qx[0], qw[0], g, g, qx[1], qw[1], bias, code, None)))
        pairs.append((ck.dequantize_nvfp4(qx[0], g, qx[1], out_dtype), ops.dequantize_nvfp4(qx[0], g, qx[1], code, True)))
    else:
        qx, qw = ck.quantize_mxfp8(x, pad_32x=True), ck.quantize_mxfp8(w)
        pairs = list(zip(qx, ops.quantize_mxfp8(x, True)))
        pairs.append((ck.scaled_mm_mxfp8(qx[0], qw[0], qx[1], qw[1], bias=bias, out_dtype=out_dtype),
                      ops.scaled_mm_mxfp8(qx[0], qw[0], qx[1], qw[1], bias, code)))
        pairs.append((ck.dequantize_mxfp8(qx[0], qx[1], out_dtype), ops.dequantize_mxfp8(qx[0], qx[1], code)))
    for a, b in pairs:
        _same(a, b)


def test_watchers_still_see_the_operator(cuda_device):
    x, _, g, _ = _operands(cuda_device)
    assert dispatcher_adds_nothing((x, g), (None,))
    with Seen() as seen:
        ck.quantize_nvfp4(x, g)
    assert any("quantize_nvfp4" in n for n in seen.names)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        ck.quantize_nvfp4(x, g)
    assert any("quantize_nvfp4" in e.name for e in prof.events())
    with torch.autograd.forward_ad.dual_level():
        assert not dispatcher_adds_nothing((x, g))
    torch.func.vmap(lambda t: (t, dispatcher_adds_nothing((x, g)) and pytest.fail("functorch is active"))[0])(x)
    assert not dispatcher_adds_nothing((x.clone().requires_grad_(), g))
    with torch.no_grad():
        assert dispatcher_adds_nothing((x.clone().requires_grad_(), g))
    assert not dispatcher_adds_nothing((x.cpu(), g)) and not dispatcher_adds_nothing((x, g), (g.cpu(),))


def test_registry_still_decides(cuda_device):
    x, _, g, _ = _operands(cuda_device)
    with pytest.raises(NoCapableBackendError):
        ck.quantize_nvfp4(x.double(), g)
    with pytest.raises(NoCapableBackendError):
        ck.quantize_mxfp8(x.reshape(2, 20, -1))
    ck.disable_backend("cuda")
    try:
        with pytest.raises(NoCapableBackendError):
            ck.quantize_nvfp4(x, g)
    finally:
        ck.enable_backend("cuda")


def test_the_registry_s_log_is_complete(cuda_device, caplog):
    x, g = torch.randn(32, 64, device=cuda_device), torch.tensor(0.01, device=cuda_device)
    with caplog.at_level("DEBUG", logger="comfy_kitchen.dispatch"):
        codes, scales = ck.quantize_nvfp4(x, g)
        ck.dequantize_nvfp4(codes, g, scales)
    assert caplog.messages == ["Backend cuda selected for quantize_nvfp4", "Backend cuda selected for dequantize_nvfp4"]


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_deterministic_mode_fills_the_outputs(cuda_device, fmt):
    x, _, g, _ = _operands(cuda_device)
    call = (lambda: ck.quantize_nvfp4(x, g)) if fmt == "nvfp4" else (lambda: ck.quantize_mxfp8(x))
    want = call()
    torch.use_deterministic_algorithms(True)
    try:
        got = call()
    finally:
        torch.use_deterministic_algorithms(False)
    for a, b in zip(want, got):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
