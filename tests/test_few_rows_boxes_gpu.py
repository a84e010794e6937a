"""Loads of an activation of fewer rows than a tile hold no more rows than there are, and half tiles from 33 rows on: what a ring slot still holds of
an earlier stage (NaN bytes of it too) must not reach a result.  Against the rows of a larger call, whose tiles have no rows left over."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# rows on both sides of 8, 16, 32, 64 and 128; half tiles, 128 x 128 tiles and splits over few and many CTAs, and a ragged last stage
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
@pytest.mark.parametrize("n, k", [(1024, 2304), (9216, 1024), (12288, 1056), (3072, 5120), (136, 4096)])
def test_same_as_rows_of_more(cuda_device, fmt, n, k):
    from comfy_kitchen.backends import cuda as backend

    mx = fmt == "mxfp8"
    gen = torch.Generator(device=cuda_device).manual_seed(n + k)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).bfloat16() for r in (128, n))
    x[127] = float("nan") if mx else 0.0
    one = torch.full((), 0.01, device=cuda_device)
    quantize = lambda t: backend.quantize_mxfp8(t) if mx else (*backend.quantize_nvfp4(t, one), one)
    qx, qw = quantize(x), quantize(w)
    mm = lambda a: (backend.scaled_mm_mxfp8(a[0], qw[0], a[1], qw[1], out_dtype=torch.float32) if mx else
                    backend.scaled_mm_nvfp4(a[0], qw[0], one, one, a[1], qw[1], out_dtype=torch.float32))
    want = mm(qx)
    for m in (1, 7, 8, 9, 16, 17, 31, 32, 33, 40, 63, 64, 65, 100, 127):
        torch.cuda.synchronize()
        mm(qx)  # leaves NaN rows (MXFP8) in shared memory
        part = quantize(x[:m].contiguous())
        got = mm(part)
        # another plan, another order of at most eight partial sums: 2^-24 an addition
        assert ((got - want[:m]).norm() / want[:m].norm()).item() <= 1e-5, m
        if not mx:
            fused = backend.linear_nvfp4_fused(part[0], qw[0], one, one, part[1], qw[1], activation="gelu_tanh", out_dtype=torch.float32) if n % 64 == 0 else None
            if fused is not None:
                ref = torch.nn.functional.gelu(want[:m], approximate="tanh")
                assert ((fused[0] - ref).norm() / ref.norm()).item() <= 1e-4, m  # the epilogue's tanh by ex2 and reciprocal
    backend.check_device_status("few rows")
