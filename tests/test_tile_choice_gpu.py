"""Which tiles a GEMM is cut into does not show in its result: the shapes on both sides of the rules against 128 x 128 tiles."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# one row block and two, half tiles that just fit 148 SMs and do not, four stages (K of NVFP4 1024, MXFP8 512) and five, a split in two
# that half tiles replace (24 stages) and one that they do not (40); 80 rows and 81 of eight stages, 80 of seven, rows of K that are no whole
# 128-byte lines in one to three row blocks; 23 stages and a split in two, columns that are no 64-byte units, 32 stages of one row block
SHAPES = [(128, 18440, 96), (129, 18440, 96), (33, 24584, 32), (65, 9216, 288), (64, 9216, 288), (66, 9536, 288), (1003, 1160, 544), (512, 9224, 1024),
          (512, 9224, 1056), (700, 3080, 512), (700, 3080, 544), (100, 9216, 24 * 128), (100, 9216, 40 * 256),
          (80, 9216, 2048), (81, 9216, 2048), (80, 9216, 1792), (68, 6304, 2976), (256, 4640, 1696), (257, 2080, 1696),
          (500, 1632, 23 * 128), (500, 1632, 23 * 256), (500, 1648, 20 * 128), (500, 1648, 20 * 256), (90, 8448, 32 * 128), (90, 8448, 32 * 256)]


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
@pytest.mark.parametrize("m, n, k", SHAPES)
def test_same_bits(cuda_device, monkeypatch, fmt, m, n, k):
    from comfy_kitchen.backends import cuda as backend

    mx = fmt == "mxfp8"
    gen = torch.Generator(device=cuda_device).manual_seed(m + n + k)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).bfloat16() for r in (m, n))
    bias = torch.linspace(-1, 1, n, device=cuda_device)
    qx, qw = ((backend.quantize_mxfp8(t) if mx else backend.quantize_nvfp4_dynamic(t)) for t in (x, w))

    def call():
        if mx:
            return backend.scaled_mm_mxfp8(qx[0], qw[0], qx[1], qw[1], bias=bias, out_dtype=torch.float32)
        return backend.scaled_mm_nvfp4(qx[0], qw[0], qx[2], qw[2], qx[1], qw[1], bias=bias, out_dtype=torch.float32)

    got = call()
    monkeypatch.setenv("CK_GEMM_CONFIG", "1")
    want = call()
    monkeypatch.delenv("CK_GEMM_CONFIG")
    if backend.load_library().ck_debug_gemm_splits(int(mx), 0, m, n, k, 1) > 1:
        assert ((got - want).norm() / want.norm()).item() <= 1e-5  # sums of K ranges in another order
    else:
        assert torch.equal(got, want)
    if not mx and n % 64 == 0:
        def fused():
            return backend.linear_nvfp4_fused(qx[0], qw[0], qx[2], qw[2], qx[1], qw[1], bias=bias, activation="gelu_tanh", requant_scale=qx[2],
                                              return_dense=False)[1:]
        got = fused()
        monkeypatch.setenv("CK_GEMM_CONFIG", "4")
        want = fused()
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, want))
    backend.check_device_status("tile choice")


@pytest.mark.parametrize("m, n, k", [(512, 6848, 768), (640, 6848, 288), (200, 4544, 768), (128, 6848, 544), (128, 7168, 544)])
def test_dynamic_linears(cuda_device, m, n, k):
    """A linear with a dynamic scale leaves SMs to the next one (54 pairs; 81, too many; half tiles on 142, 107 and 112 SMs): the bits of
    the separate calls, several in a row."""
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(m + n)
    w, bias = torch.randn(n, k, generator=gen, device=cuda_device).bfloat16(), torch.linspace(-1, 1, n, device=cuda_device)
    qw = backend.quantize_nvfp4_dynamic(w)
    xs = [torch.randn(m, k, generator=gen, device=cuda_device).bfloat16() * s for s in (1, 20, 0.3)]
    got = [backend.linear_nvfp4_from_float(x, qw[0], qw[2], qw[1], bias=bias) for x in xs]
    for x, y in zip(xs, got):
        q, s, g = backend.quantize_nvfp4_dynamic(x)
        assert torch.equal(y, backend.scaled_mm_nvfp4(q, qw[0], g, qw[2], s, qw[1], bias=bias))
    backend.check_device_status("dynamic linears")
