"""Loads of an activation of fewer rows than a tile hold no more rows than there are, and half tiles from 33 rows on: what a ring slot still
holds of an earlier kernel, and what the scale tensor holds in its padding rows, must not reach a result.  Every call stands directly behind one of
128 rows of extreme values, and the scales of its padding rows are NaN, so that every accumulator row past the last one is."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = (1, 7, 8, 9, 16, 17, 31, 32, 33, 40, 63, 64, 65, 100, 127)


def _poisoned(scales, m, nan):
    """The tiled scales of 128 rows (tiles of 32 x 4 x 4 bytes) with NaN in those from m on."""
    bad = scales.clone()
    tiles = bad.view(torch.uint8).view(-1, 32, 4, 4)
    for r in range(m, 128):
        tiles[:, r % 32, r // 32] = nan
    return bad


# rows on both sides of 8, 16, 32, 64 and 128; half tiles, 128 x 128 tiles and splits over few and many CTAs, and a ragged last stage; the kernel that
# the size takes, 128 x 128 tiles and half tiles (the call before goes through the same kernel there)
@pytest.mark.parametrize("config", [None, "1", "7"])
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
@pytest.mark.parametrize("n, k", [(1024, 2304), (9216, 1024), (12288, 1056), (3072, 5120), (136, 4096)])
def test_rows_past_the_last_one(cuda_device, monkeypatch, fmt, n, k, config):
    from comfy_kitchen.backends import cuda as backend

    mx = fmt == "mxfp8"
    gen = torch.Generator(device=cuda_device).manual_seed(n + k)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).bfloat16() for r in (128, n))
    one = torch.full((), 0.01, device=cuda_device)
    quantize = lambda t: backend.quantize_mxfp8(t) if mx else backend.quantize_nvfp4(t, one)
    qx, qw = quantize(x), quantize(w)
    extreme = quantize(torch.full_like(x, float("nan") if mx else 3e4))
    parts = {m: quantize(x[:m].contiguous()) for m in ROWS}
    bad = {m: (codes, _poisoned(scales, m, 0xFF if mx else 0x7F)) for m, (codes, scales) in parts.items()}
    if config is not None:
        monkeypatch.setenv("CK_GEMM_CONFIG", config)

    def mm(a):
        if mx:
            return backend.scaled_mm_mxfp8(a[0], qw[0], a[1], qw[1], out_dtype=torch.float32)
        return backend.scaled_mm_nvfp4(a[0], qw[0], one, one, a[1], qw[1], out_dtype=torch.float32)

    want = mm(qx)
    for m in ROWS:
        torch.cuda.synchronize()
        mm(extreme)
        got = mm(bad[m])
        clean = mm(parts[m])
        # another plan than that of 128 rows, another order of at most eight partial sums: 2^-24 an addition
        assert torch.equal(got, clean) and ((got - want[:m]).norm() / want[:m].norm()).item() <= 1e-5, m
        # the poison is where it should be: one row further down it takes the last row, all of it and no other
        lost = mm((bad[m][0], _poisoned(parts[m][1], m - 1, 0xFF if mx else 0x7F))).isnan()
        assert lost[m - 1].all() and not lost[: m - 1].any(), m
    backend.check_device_status("few rows")


@pytest.mark.parametrize("config", [None, "1"])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n, k", [(1024, 2304), (9216, 1056)])
def test_padding_rows_of_the_fused_epilogue(cuda_device, monkeypatch, n, k, out_dtype, config):
    """Rows past the last one are padding of the re-quantized scales: zeros, whatever their accumulators hold."""
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(n + k)
    x, w = (torch.randn(r, k, generator=gen, device=cuda_device).bfloat16() for r in (128, n))
    one = torch.full((), 0.01, device=cuda_device)
    qw = backend.quantize_nvfp4(w, one)
    extreme = backend.quantize_nvfp4(torch.full_like(x, 3e4), one)
    parts = {m: backend.quantize_nvfp4(x[:m].contiguous(), one) for m in ROWS}
    bad = {m: (codes, _poisoned(scales, m, 0x7F)) for m, (codes, scales) in parts.items()}
    if config is not None:
        monkeypatch.setenv("CK_GEMM_CONFIG", config)
    rq = torch.full((), 0.05, device=cuda_device)
    fused = lambda a, activation, dense: backend.linear_nvfp4_fused(a[0], qw[0], one, one, a[1], qw[1], activation=activation, out_dtype=out_dtype,
                                                                    requant_scale=rq, return_dense=dense)
    for m in ROWS:
        for activation, dense in ((None, True), ("gelu_tanh", True), ("gelu_tanh", False)):
            torch.cuda.synchronize()
            fused(extreme, activation, dense)
            got = fused(bad[m], activation, dense)
            hidden = fused(parts[m], activation, True)[0]
            codes, scales = backend.quantize_nvfp4(hidden, rq)
            assert not dense or torch.equal(got[0], hidden), m
            assert torch.equal(got[1], codes) and torch.equal(got[2].view(torch.uint8).flatten(), scales.view(torch.uint8).flatten()), m
    backend.check_device_status("few rows")
