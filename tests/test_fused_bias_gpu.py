"""Bias of the fused epilogue, staged by each warp for itself: several tiles to a worker (74 pairs, 148 single CTAs), two accumulators, ragged rows
and columns, every bias type, against the separate calls."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.float16, torch.bfloat16, None])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
# pairs: 85 and 297 tiles, the last columns 64 and 192 wide; 128 x 128: 153 and 650 tiles; one tile to a CTA
@pytest.mark.parametrize("m, n, k, config", [(1100, 4160, 288, None), (2100, 8384, 64, None), (300, 6464, 96, "1"), (1200, 8256, 544, "1"), (130, 320, 64, None)])
def test_bias_of_many_tiles(cuda_device, monkeypatch, m, n, k, config, dtype, bias_dtype):
    import comfy_kitchen as ck
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(m + n + k)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).bfloat16() for r in (m, n))
    bias = None if bias_dtype is None else (torch.randn(n, generator=gen, device=cuda_device) * 4).to(bias_dtype)
    (qx, sx, gx), (qw, sw, gw) = backend.quantize_nvfp4_dynamic(x), backend.quantize_nvfp4_dynamic(w)
    scale = torch.full((), 0.02, device=cuda_device)
    want = ck.scaled_mm_nvfp4(qx, qw, gx, gw, sx, sw, bias=bias, out_dtype=dtype)
    want_codes, want_scales = backend.quantize_nvfp4(want, scale)
    if config is not None:
        monkeypatch.setenv("CK_GEMM_CONFIG", config)
    fused = lambda **kw: backend.linear_nvfp4_fused(qx, qw, gx, gw, sx, sw, bias=bias, out_dtype=dtype, requant_scale=scale, **kw)
    dense, codes, scales = fused(activation=None)
    assert torch.equal(dense, want)
    assert torch.equal(codes, want_codes[:m]) and torch.equal(scales.view(torch.uint8).flatten(), want_scales.view(torch.uint8).flatten())
    _, with_dense, scales_with = fused(activation="gelu_tanh")
    _, alone, scales_alone = fused(activation="gelu_tanh", return_dense=False)  # the straight path
    assert torch.equal(with_dense, alone) and torch.equal(scales_with.view(torch.uint8), scales_alone.view(torch.uint8))
    backend.check_device_status("fused bias")
