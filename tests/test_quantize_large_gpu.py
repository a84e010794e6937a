"""The dynamic quantizer on inputs of more chunks than there are partial maxima, and of sizes on both sides of
the rules that go by the input's bytes: the same bits as in parts, with the scale of the whole."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# 2100 x 4096 fp32 is 33 MiB, 1050 chunks; 88000 x 3072 bf16 is 516 MiB, more than 16384 chunks of 32 KiB
@pytest.mark.parametrize("rows, cols, dtype", [(2100, 4096, torch.float32), (7300, 3072, torch.bfloat16), (88000, 3072, torch.bfloat16)])
@pytest.mark.parametrize("where", ["first", "last", "middle"])
def test_large_input_equals_its_parts(cuda_device, rows, cols, dtype, where):
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device, dtype=torch.float32).to(dtype)
    flat = x.view(-1)
    flat[{"first": 0, "last": -1, "middle": flat.numel() // 2 + 77}[where]] = -1000.0
    codes, block_scales, scale = backend.quantize_nvfp4_dynamic(x)
    assert torch.equal(scale, (torch.tensor(1000.0, dtype=dtype, device=cuda_device) / 2688.0).float())
    for start in range(0, rows, 1024):  # multiples of 128 rows: whole scale tiles
        part = x[start:start + 1024]
        want_codes, want_scales = backend.quantize_nvfp4(part.contiguous(), scale)
        assert torch.equal(codes[start:start + 1024], want_codes)
        tiles = want_scales.view(torch.uint8).flatten()
        at = start * block_scales.shape[1]
        assert torch.equal(block_scales.view(torch.uint8).flatten()[at:at + tiles.numel()], tiles)
