"""A kernel that somebody registers for an operator of this package is the one that ``ck.*`` calls."""
from __future__ import annotations

import pytest
import torch

import comfy_kitchen as ck
from comfy_kitchen import ops

OPERATORS = ["quantize_nvfp4", "dequantize_nvfp4", "scaled_mm_nvfp4", "quantize_mxfp8", "dequantize_mxfp8", "scaled_mm_mxfp8"]


@pytest.mark.parametrize("name", OPERATORS)
def test_registrations_are_seen_and_their_removal(name):
    assert not ops.replaced(name)
    for key in ("CUDA", "AutocastCUDA", "AutogradCUDA"):
        lib = torch.library.Library("comfy_kitchen", "FRAGMENT")
        lib.impl(name, lambda *args: None, key)
        assert ops.replaced(name)
        assert not any(ops.replaced(other) for other in OPERATORS if other != name)
        lib._destroy()
        assert not ops.replaced(name)


def test_another_package_s_registration_is_not_ours():
    lib = torch.library.Library("ck_test_other", "DEF")
    lib.define("quantize_nvfp4(Tensor x) -> Tensor")
    lib.impl("quantize_nvfp4", lambda x: x, "CUDA")
    assert not ops.replaced("quantize_nvfp4")
    lib._destroy()


def test_kernel_for_all_devices_is_seen():
    kernels = ops._op_quantize_mxfp8._backend_fns
    before = dict(kernels)
    try:
        kernels[None] = lambda x, pad_32x: None  # what register_kernel for all devices leaves
        assert ops.replaced("quantize_mxfp8")
    finally:
        kernels.clear()
        kernels.update(before)
    assert not ops.replaced("quantize_mxfp8")


@pytest.mark.gpu
def test_replacement_is_called(cuda_device):
    x, g = torch.ones(16, 32, device=cuda_device, dtype=torch.bfloat16), torch.tensor(0.01, device=cuda_device)
    codes, scales = ck.quantize_nvfp4(x, g)
    lib = torch.library.Library("comfy_kitchen", "FRAGMENT")
    try:
        lib.impl("quantize_nvfp4", lambda x, scale, eps, pad, hi: (torch.full_like(codes, 7), scales.clone()), "CUDA")
        assert torch.equal(ck.quantize_nvfp4(x, g)[0], torch.full_like(codes, 7))
    finally:
        lib._destroy()
    assert torch.equal(ck.quantize_nvfp4(x, g)[0], codes)


def test_the_native_half_steps_aside_for_a_replaced_function(monkeypatch):
    import types

    from comfy_kitchen.backends import cuda as backend

    names = [*OPERATORS, "quantize_nvfp4_dynamic"]
    monkeypatch.setattr(backend, "_host", types.SimpleNamespace(**{name: name for name in names}))
    for name in names:
        assert backend.host_function(name) == name
        with monkeypatch.context() as m:
            m.setattr(backend, name, lambda *args, **kwargs: None)
            assert backend.host_function(name) is None
            assert all(backend.host_function(other) == other for other in names if other != name)
        assert backend.host_function(name) == name
