"""fp32 inputs larger than L2 are quantized from their last rows on when the scale comes from a reduction: the same bits as with that
scale given, on both sides of both lines (120 MiB of input, 64 MiB of codes and scales), with rows and columns that end inside a block and
padded rows.  Which inputs they are: test_quantize_walk_cpu."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# 10240 x 3072 fp32 is 120 MiB; 38900 x 3072 has more than 64 MiB of codes and scales (no marks, forwards)
@pytest.mark.parametrize("rows, cols, pad", [(10240, 3072, False), (10241, 3072, True), (10255, 3088, False), (20001, 1584, True), (130, 262144, False), (38900, 3072, False)])
def test_same_as_with_the_scale_given(cuda_device, rows, cols, pad):
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device)
    x[0, 0], x[rows // 2, cols - 1] = -77.0, 900.0
    codes, block_scales, scale = backend.quantize_nvfp4_dynamic(x, pad_16x=pad)
    assert scale.item() == (torch.tensor(900.0, device=cuda_device) / 2688.0).item()
    want_codes, want_scales = backend.quantize_nvfp4(x, scale, pad_16x=pad)
    assert torch.equal(codes, want_codes) and torch.equal(block_scales.view(torch.uint8), want_scales.view(torch.uint8))
