"""Dynamic scales on both sides of the sizes up to which the quantizer's blocks (more than eight rows 128 KiB, else 64) and the few-row linear's CTAs
(128 KiB; where two share an SM 64, fp32 112) take the maximum of the whole input themselves: the bits of the scale on its own and of the separate calls, whichever element is the largest."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [1, 8, 9, 33, 130])
@pytest.mark.parametrize("kib", [64, 128])
@pytest.mark.parametrize("where", ["first", "middle", "last", "nan"])
def test_scale_and_codes(cuda_device, dtype, rows, kib, where):
    from comfy_kitchen.backends import cuda as backend

    elem = torch.empty((), dtype=dtype).element_size()
    line = (kib << 10) // elem // rows // 32 * 32  # the most columns that stay within it
    gen = torch.Generator(device=cuda_device).manual_seed(rows + kib)
    for k in (line, line + 32):
        x = torch.randn(rows, k, generator=gen, device=cuda_device).to(dtype)
        at = {"first": 0, "middle": x.numel() // 2 + 5, "last": x.numel() - 1, "nan": 7}[where]
        x.view(-1)[at] = float("nan") if where == "nan" else -50.0
        scale = backend.nvfp4_tensor_scale(x)
        if where != "nan":
            want = (x.abs().amax() / 2688).float()  # the division in the input's type
            assert torch.equal(scale, want)
        codes, block_scales, got = backend.quantize_nvfp4_dynamic(x)
        assert torch.equal(got, scale)
        want_codes, want_scales = backend.quantize_nvfp4(x, scale)
        assert torch.equal(codes, want_codes) and torch.equal(block_scales.view(torch.uint8), want_scales.view(torch.uint8))
        if where == "nan":
            continue
        w = torch.randn(256, k, generator=gen, device=cuda_device).bfloat16()
        qw, sw, gw = backend.quantize_nvfp4_dynamic(w)
        got = backend.linear_nvfp4_from_float(x, qw, gw, sw, out_dtype=torch.float32)
        want = backend.scaled_mm_nvfp4(codes, qw, scale, gw, block_scales, sw, out_dtype=torch.float32)
        assert torch.equal(got, want)


# a weight of more 128-row tiles than SMs, or so long a K that a tile's clusters share SMs
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows, n, kib", [(8, 19072, 64), (8, 19072, 112), (1, 4096, 64), (2, 4096, 112), (2, 4096, 128)])
def test_two_ctas_to_an_sm(cuda_device, dtype, rows, n, kib):
    from comfy_kitchen.backends import cuda as backend

    elem = torch.empty((), dtype=dtype).element_size()
    line = (kib << 10) // elem // rows // 32 * 32
    gen = torch.Generator(device=cuda_device).manual_seed(rows + n)
    for k in (line, line + 32):
        x = torch.randn(rows, k, generator=gen, device=cuda_device).to(dtype)
        x.view(-1)[-1] = -50.0
        qw, sw, gw = backend.quantize_nvfp4_dynamic(torch.randn(n, k, generator=gen, device=cuda_device, dtype=torch.bfloat16))
        scale = backend.nvfp4_tensor_scale(x)
        codes, block_scales = backend.quantize_nvfp4(x, scale)
        got = backend.linear_nvfp4_from_float(x, qw, gw, sw, out_dtype=torch.float32)
        assert torch.equal(got, backend.scaled_mm_nvfp4(codes, qw, scale, gw, block_scales, sw, out_dtype=torch.float32))
    backend.check_device_status("whole input")
