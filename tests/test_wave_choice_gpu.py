"""128 x 128 tiles instead of pairs where they take no more waves, half tiles instead of a split in two up to 36 stages: sizes on both sides of
the lines (148 SMs) against forced 128 x 128 tiles, plain, fused and behind a dynamic quantizer."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# one wave of tiles and of pairs: 144 tiles of three row blocks; 147 and 150 tiles; two waves of either, and three against two; padded rows; 36 and
# 37 stages of half tiles, and columns that rule them out; one wave more at the last stages it is taken for and one beyond, rows that straddle lines
SHAPES = [(300, 6144, 1312), (257, 6272, 1312), (257, 6400, 1312), (384, 12288, 1312), (384, 12672, 1312), (1152, 4096, 1344), (700, 3520, 1312),
          (512, 9216, 6 * 128), (512, 9216, 6 * 256), (512, 9216, 7 * 256), (700, 6144, 5 * 256 - 32), (1100, 4608, 5 * 128), (1100, 4608, 6 * 256), (1152, 7680, 5 * 256),
          (512, 9216, 12 * 256), (512, 9216, 2 * 256), (1100, 4608, 13 * 256), (256, 4608, 36 * 128), (256, 4608, 37 * 128), (256, 4608, 36 * 256), (256, 4608, 37 * 256 - 32), (256, 4616, 30 * 128)]


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
@pytest.mark.parametrize("m, n, k", SHAPES)
def test_same_as_128_x_128(cuda_device, monkeypatch, fmt, m, n, k):
    from comfy_kitchen.backends import cuda as backend

    mx = fmt == "mxfp8"
    gen = torch.Generator(device=cuda_device).manual_seed(m + n + k)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).bfloat16() for r in (m, n))
    bias = torch.linspace(-1, 1, n, device=cuda_device)
    qx, qw = ((backend.quantize_mxfp8(t) if mx else backend.quantize_nvfp4_dynamic(t)) for t in (x, w))

    def calls():
        if mx:
            return backend.scaled_mm_mxfp8(qx[0], qw[0], qx[1], qw[1], bias=bias, out_dtype=torch.float32), backend.linear_mxfp8_from_float(
                x, qw[0], qw[1], bias=bias, out_dtype=torch.float32)
        fused = ()
        if n % 64 == 0:
            fused = backend.linear_nvfp4_fused(qx[0], qw[0], qx[2], qw[2], qx[1], qw[1], bias=bias, activation="gelu_tanh", requant_scale=qx[2],
                                               return_dense=False)[1:]
        return (backend.scaled_mm_nvfp4(qx[0], qw[0], qx[2], qw[2], qx[1], qw[1], bias=bias, out_dtype=torch.float32),
                backend.linear_nvfp4_from_float(x, qw[0], qw[2], qw[1], bias=bias, out_dtype=torch.float32), *fused)

    got = calls()
    monkeypatch.setenv("CK_GEMM_CONFIG", "1")
    want = calls()
    monkeypatch.delenv("CK_GEMM_CONFIG")
    split = backend.load_library().ck_debug_gemm_splits(int(mx), 0, m, n, k, 0) > 1 or backend.load_library().ck_debug_gemm_splits(int(mx), 0, m, n, k, 1) > 1
    for a, b in zip(got, want):
        if split and a.dtype == torch.float32:
            assert ((a - b).norm() / b.norm()).item() <= 1e-5  # sums of K ranges in another order: 2^-24 an addition
        else:
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    backend.check_device_status("wave choice")


# fused in fp32: pairs where they take one wave and 128 x 128 tiles two; three waves of those against two up to twelve stages
@pytest.mark.parametrize("m, n, k", [(1024, 4608, 4 * 256), (384, 9216, 256 + 32), (1000, 4672, 5 * 256), (1152, 4608, 12 * 256), (1152, 4608, 13 * 256)])
def test_fused_fp32_same_as_128_x_128(cuda_device, monkeypatch, m, n, k):
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(m + n + k)
    (qx, sx, gx), (qw, sw, gw) = (backend.quantize_nvfp4_dynamic(torch.randn(r, k, generator=gen, device=cuda_device).bfloat16()) for r in (m, n))
    bias = torch.linspace(-1, 1, n, device=cuda_device)
    call = lambda dense: backend.linear_nvfp4_fused(qx, qw, gx, gw, sx, sw, bias=bias, activation="gelu_tanh", out_dtype=torch.float32,
                                                    requant_scale=gx, return_dense=dense)
    got, got_alone = call(True), call(False)
    monkeypatch.setenv("CK_GEMM_CONFIG", "1")
    want = call(True)
    for a, b, c in zip(want, got, (want[0], *got_alone[1:])):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)) and torch.equal(a.view(torch.uint8), c.view(torch.uint8))
    backend.check_device_status("fused in fp32")
