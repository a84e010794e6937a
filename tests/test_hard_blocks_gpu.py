"""Blocks that the straight NVFP4 code cannot settle (operands on rounding boundaries, scales outside its window, mixed
with ordinary and zero blocks) against the build of the quantizer that divides every element."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _hard(rows, cols, g, dtype, device):
    gen = torch.Generator(device=device).manual_seed(7)
    x = torch.randn(rows, cols // 16, 16, generator=gen, device=device)
    kind = torch.randint(0, 5, (rows, cols // 16, 1), generator=gen, device=device)
    middles = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0], device=device)
    on = middles[torch.randint(0, 8, x.shape, generator=gen, device=device)] * torch.sign(x)
    on[..., 0] = 6.0
    # total scale = g * s for s exact in E4M3: x / total lies on the middles; a nudge of one ulp on some
    s = 2.0 ** torch.randint(-3, 6, kind.shape, generator=gen, device=device) * 1.125
    tie = (on * s * g).float()
    nudged = torch.nextafter(tie, torch.full_like(tie, float("inf")))
    edge = x * s * g  # the block's own scale next to a boundary of E4M3: amax = 6 g (s + half a step)
    edge[..., 3:4] = 6.0 * g * (s + s / 1.125 / 16)
    x = torch.where(kind == 0, tie, torch.where(kind == 1, nudged, torch.where(kind == 2, edge, torch.where(kind == 3, x * g, torch.zeros_like(x)))))
    return x.reshape(rows, cols).to(dtype).contiguous()


@pytest.mark.parametrize("g", [0.0078125, 2.0 ** -45, 2.0 ** 44, 0.0031])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [8, 1024])
def test_same_as_dividing(cuda_device, rows, dtype, g):
    if dtype == torch.float16 and not 1e-4 < g < 1:
        pytest.skip("outside of float16")
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    scale = torch.tensor(g, dtype=torch.float32, device=cuda_device)
    x = _hard(rows, 1024, g, dtype, cuda_device)
    codes, blocks = backend.quantize_nvfp4(x, scale)
    before = lib.ck_debug_set_exact_division(1)
    try:
        ref_codes, ref_blocks = backend.quantize_nvfp4(x, scale)
    finally:
        lib.ck_debug_set_exact_division(before)
    assert torch.equal(codes, ref_codes) and torch.equal(blocks.view(torch.uint8), ref_blocks.view(torch.uint8))
    if rows == 8:  # the linear of few rows quantizes these rows itself
        one = torch.tensor(2.0 ** -20, device=cuda_device)
        w, w_blocks = backend.quantize_nvfp4(torch.randn(136, 1024, device=cuda_device).bfloat16() * 1e-4, one)
        got = backend.linear_nvfp4_from_float(x, w, one, w_blocks, x_scale=scale, out_dtype=torch.float32)
        ref = backend.scaled_mm_nvfp4(ref_codes, w, scale, one, ref_blocks, w_blocks, out_dtype=torch.float32)
        assert torch.equal(got, ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_fused_epilogue(cuda_device, dtype):
    """GELU and re-quantization in the epilogue against GELU's dense result, divided: a hidden scale that puts many of its
    16-bit values on boundaries (a power of two), one outside the window, and rows and columns that end inside a tile."""
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    m, n, k = 300, 576, 256
    gen = torch.Generator(device=cuda_device).manual_seed(8)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).to(dtype) for r in (m, n))
    qx, qw = backend.quantize_nvfp4_dynamic(x), backend.quantize_nvfp4_dynamic(w)
    for g in (2.0 ** -5, 0.01, 2.0 ** -44):
        rq = torch.tensor(g, dtype=torch.float32, device=cuda_device)

        def call(dense):
            return backend.linear_nvfp4_fused(qx[0], qw[0], qx[2], qw[2], qx[1], qw[1], activation="gelu_tanh", out_dtype=dtype,
                                              requant_scale=rq, return_dense=dense)

        h, codes, blocks = call(True)
        _, only_codes, only_blocks = call(False)
        before = lib.ck_debug_set_exact_division(1)
        try:
            ref_codes, ref_blocks = backend.quantize_nvfp4(h, rq)
        finally:
            lib.ck_debug_set_exact_division(before)
        for c, b in ((codes, blocks), (only_codes, only_blocks)):
            assert torch.equal(c, ref_codes) and torch.equal(b.view(torch.uint8), ref_blocks.view(torch.uint8))
