"""The dynamic quantizer on inputs of more chunks than there are partial maxima, and of sizes on both sides of
the rules that go by the input's bytes: the same bits as in parts, with the scale of the whole."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# 2100 x 4096 fp32 is 33 MiB in 525 chunks; 38900 x 3072 has 64.1 MiB of codes and scales; 88000 x 3072 bf16 is 516 MiB, more than 16384 chunks of 32 KiB
@pytest.mark.parametrize("rows, cols, dtype", [(2100, 4096, torch.float32), (7300, 3072, torch.bfloat16), (38900, 3072, torch.bfloat16), (88000, 3072, torch.bfloat16)])
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


# padded rows x columns on both sides of the line between the two kernels of small fp32 inputs, and padded rows
@pytest.mark.parametrize("rows, cols", [(1, 16), (128, 5104), (128, 5120), (100, 5120), (33, 5136), (640, 1008), (640, 1024), (7, 48)])
def test_fp32_kernels_agree(cuda_device, rows, cols):
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device, dtype=torch.float32)
    want_codes, want_scales, scale = backend.quantize_nvfp4_dynamic(x)  # streams at every size
    codes, block_scales = backend.quantize_nvfp4(x, scale)
    assert torch.equal(codes, want_codes) and torch.equal(block_scales.view(torch.uint8), want_scales.view(torch.uint8))
    padded, padded_scales = backend.quantize_nvfp4(x, scale, pad_16x=True)
    assert torch.equal(padded[:rows], codes) and not padded[rows:].any()
    assert torch.equal(padded_scales.view(torch.uint8), block_scales.view(torch.uint8))


# on both sides of the lines between blocks of 4 and 16 rows, resident or two passes each, with rows and columns that end inside a block
@pytest.mark.parametrize("rows, cols, dtype", [(128, 3072, torch.bfloat16), (777, 3072, torch.float16), (896, 3072, torch.bfloat16), (1, 64, torch.bfloat16),
                                               (6145, 6208, torch.bfloat16), (6143, 6208, torch.float16), (12288, 3104, torch.bfloat16),
                                               (3100, 6400, torch.float32), (25000, 3088, torch.float32), (18000, 3072, torch.float32)])
@pytest.mark.parametrize("hi_first", [True, False])
def test_block_shapes_of_the_static_quantizer(cuda_device, rows, cols, dtype, hi_first):
    """Against the build of the quantizer that divides every element, whose kernel has one block shape."""
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device, dtype=torch.float32).to(dtype)
    g = torch.tensor(0.0021, device=cuda_device)
    got = backend.quantize_nvfp4(x, g, hi_first=hi_first)
    before = lib.ck_debug_set_exact_division(1)
    try:
        want = backend.quantize_nvfp4(x, g, hi_first=hi_first)
    finally:
        lib.ck_debug_set_exact_division(before)
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
