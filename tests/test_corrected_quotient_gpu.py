"""Codes of 16-bit inputs by the corrected quotient (stand-alone quantizer, few-row linear) against the build that divides every element:
every finite bit pattern, and blocks on rounding boundaries under a tensor scale whose significand is all ones."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

ALL_ONES = 2.0 ** -7 * (1 - 2.0 ** -24)


def _patterns(dtype, device):
    """All finite patterns, 15 in a block behind one that fixes the block's maximum."""
    bits = torch.arange(65536, device=device, dtype=torch.int32).to(torch.int16).view(dtype)
    bits = bits[torch.isfinite(bits)]
    bits = bits[: bits.numel() // 15 * 15].view(-1, 15)
    top = 2.0 ** (torch.arange(bits.shape[0], device=device) % 12 - 3) * 1.625
    top = torch.maximum(top, bits.float().abs().amax(1)).to(dtype)
    return torch.cat([top.unsqueeze(1), bits], 1)


def _on_boundaries(dtype, device):
    gen = torch.Generator(device=device).manual_seed(3)
    middles = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0], device=device)
    x = middles[torch.randint(0, 8, (4096, 16), generator=gen, device=device)] * (torch.randint(0, 2, (4096, 16), generator=gen, device=device) * 2 - 1)
    x[:, 0] = 6.0
    return (x * 2.0 ** -7 * 2.0 ** torch.randint(-2, 5, (4096, 1), generator=gen, device=device)).to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("g", [ALL_ONES, 2.0 ** -7, 0.0031])
def test_same_as_dividing(cuda_device, dtype, g):
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    scale = torch.tensor(g, dtype=torch.float32, device=cuda_device)
    blocks = torch.cat([_patterns(dtype, cuda_device), _on_boundaries(dtype, cuda_device)])
    blocks = blocks[: blocks.shape[0] // 32 * 32].reshape(-1, 512).contiguous()
    codes, scales = backend.quantize_nvfp4(blocks, scale)
    before = lib.ck_debug_set_exact_division(1)
    try:
        ref_codes, ref_scales = backend.quantize_nvfp4(blocks, scale)
        x = blocks[-8:].contiguous()
        ref_x = backend.quantize_nvfp4(x, scale)
    finally:
        lib.ck_debug_set_exact_division(before)
    assert torch.equal(codes, ref_codes) and torch.equal(scales.view(torch.uint8), ref_scales.view(torch.uint8))
    one = torch.tensor(2.0 ** -20, device=cuda_device)
    w, w_scales = backend.quantize_nvfp4(torch.randn(136, 512, device=cuda_device).bfloat16() * 1e-4, one)
    got = backend.linear_nvfp4_from_float(x, w, one, w_scales, x_scale=scale, out_dtype=torch.float32)
    ref = backend.scaled_mm_nvfp4(ref_x[0], w, scale, one, ref_x[1], w_scales, out_dtype=torch.float32)
    assert torch.equal(got, ref)
