"""One-call linears of up to 16 rows quantize the activation inside the GEMM: the bits of the separate calls."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# rows (the last that are quantized inside, and the first that are not), ragged weights, K of less than a stage, with a short last
# stage or an odd number of 32-element blocks, K over clusters of 4 to 8 CTAs, more tiles than SMs, x of 128 KiB in 16 bits
# and beyond (a reduction kernel)
SHAPES = [(1, 8, 32), (1, 1040, 96), (2, 136, 288), (3, 264, 1056), (4, 18432, 64), (5, 136, 24 * 256 - 32), (7, 520, 544), (8, 128, 256),
          (8, 19200, 96), (8, 3072, 6112), (9, 264, 544), (8, 1024, 8192), (8, 1024, 8224), (12, 128, 1120), (16, 264, 4064), (16, 128, 32), (17, 136, 288)]


def _x(m, k, dtype, device, seed):
    gen = torch.Generator(device=device).manual_seed(seed)
    x = torch.randn(m, k, generator=gen, device=device)
    x[:, ::37] *= 40
    x[m // 2, : k // 2] = 0  # whole blocks of zeros
    return x.to(dtype)


def _w(n, k, device):
    gen = torch.Generator(device=device).manual_seed(n + k)
    return (torch.randn(n, k, generator=gen, device=device) * 0.02).bfloat16(), torch.linspace(-1, 1, n, device=device)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m, n, k", SHAPES)
@pytest.mark.parametrize("fmt", ["nvfp4", "nvfp4_static", "mxfp8"])
def test_same_bits_as_the_separate_calls(cuda_device, fmt, m, n, k, dtype):
    from comfy_kitchen.backends import cuda as backend

    w, bias = _w(n, k, cuda_device)
    out_dtype = {8: torch.float32, 3: torch.float16}.get(m, torch.bfloat16)
    qw = backend.quantize_mxfp8(w) if fmt == "mxfp8" else backend.quantize_nvfp4_dynamic(w)
    for seed in (1, 2):  # one call right behind another, on other data
        x = _x(m, k, dtype, cuda_device, seed)
        if fmt == "mxfp8":
            got = backend.linear_mxfp8_from_float(x, *qw, bias=bias, out_dtype=out_dtype)
            q, s = backend.quantize_mxfp8(x)
            ref = backend.scaled_mm_mxfp8(q, qw[0], s, qw[1], bias=bias, out_dtype=out_dtype)
        else:
            g = backend.nvfp4_tensor_scale(x)
            got = backend.linear_nvfp4_from_float(x, qw[0], qw[2], qw[1], bias=bias, x_scale=g if fmt == "nvfp4_static" else None,
                                                  out_dtype=out_dtype)
            q, s = backend.quantize_nvfp4(x, g)
            ref = backend.scaled_mm_nvfp4(q, qw[0], g, qw[2], s, qw[1], bias=bias, out_dtype=out_dtype)
        assert torch.isfinite(ref).all() and torch.equal(got, ref)
    backend.check_device_status("linear of few rows")


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_other_routes_for_the_same_rows(cuda_device, fmt):
    """A misaligned activation and the validation hook of the quantizers go through the separate kernels."""
    from comfy_kitchen.backends import cuda as backend

    w, bias = _w(136, 288, cuda_device)
    qw = backend.quantize_mxfp8(w) if fmt == "mxfp8" else backend.quantize_nvfp4_dynamic(w)

    def call(x):
        if fmt == "mxfp8":
            return backend.linear_mxfp8_from_float(x, *qw, bias=bias)
        return backend.linear_nvfp4_from_float(x, qw[0], qw[2], qw[1], bias=bias)

    x = _x(4, 288, torch.bfloat16, cuda_device, 3)
    want = call(x)
    shifted = torch.empty(4 * 288 + 8, dtype=x.dtype, device=cuda_device)[8:].view(4, 288)
    shifted.copy_(x)
    assert shifted.data_ptr() % 32 != 0 and torch.equal(call(shifted), want)
    lib = backend.load_library()
    before = lib.ck_debug_set_exact_division(1)
    try:
        assert torch.equal(call(x), want)
    finally:
        lib.ck_debug_set_exact_division(before)


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_result_over_the_activation(cuda_device, fmt):
    """The C entry points write a result over the activation it came from; results right beside it don't count."""
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    m, n, k = 4, 288, 576
    w, _ = _w(n, k, cuda_device)
    x = _x(m, k, torch.bfloat16, cuda_device, 4)
    stream = torch.cuda.current_stream().cuda_stream
    bf16 = 2
    if fmt == "mxfp8":
        q, s = backend.quantize_mxfp8(w)
        size = lib.ck_linear_mxfp8_from_float_workspace_bytes(m, k)
        want = backend.linear_mxfp8_from_float(x, q, s)
    else:
        q, s, g = backend.quantize_nvfp4_dynamic(w)
        size = lib.ck_linear_nvfp4_from_float_workspace_bytes(m, k, 1)
        want = backend.linear_nvfp4_from_float(x, q, g, s)
    ws = torch.empty(size, dtype=torch.uint8, device=cuda_device)
    for offset in (0, m * k - 16, m * k):  # in elements: over it, over its last bytes, behind it
        buf = torch.empty(m * k + m * n, dtype=x.dtype, device=cuda_device)
        buf[: m * k].copy_(x.flatten())
        out = buf[offset : offset + m * n]
        if fmt == "mxfp8":
            rc = lib.ck_linear_mxfp8_from_float(buf.data_ptr(), bf16, q.data_ptr(), s.data_ptr(), None, 0, out.data_ptr(), bf16, m, n, k,
                                                ws.data_ptr(), size, stream)
        else:
            rc = lib.ck_linear_nvfp4_from_float(buf.data_ptr(), bf16, None, q.data_ptr(), s.data_ptr(), g.data_ptr(), None, 0, out.data_ptr(),
                                                bf16, m, n, k, ws.data_ptr(), size, stream)
        assert rc == 0 and torch.equal(out.view(m, n), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("fmt", ["nvfp4", "nvfp4_static", "mxfp8"])
def test_infinities_and_nan(cuda_device, fmt, value, dtype):
    from comfy_kitchen.backends import cuda as backend

    m, n, k = 5, 136, 608
    w, bias = _w(n, k, cuda_device)
    x = _x(m, k, dtype, cuda_device, 5)
    g = backend.nvfp4_tensor_scale(x)
    x[1, 3], x[3, k - 1], x[3, 40] = value, value, float("inf")
    if fmt == "mxfp8":
        qw = backend.quantize_mxfp8(w)
        got = backend.linear_mxfp8_from_float(x, *qw, bias=bias, out_dtype=torch.bfloat16)
        q, s = backend.quantize_mxfp8(x)
        ref = backend.scaled_mm_mxfp8(q, qw[0], s, qw[1], bias=bias, out_dtype=torch.bfloat16)
    else:
        qw = backend.quantize_nvfp4_dynamic(w)
        if fmt == "nvfp4":
            g = backend.nvfp4_tensor_scale(x)
        got = backend.linear_nvfp4_from_float(x, qw[0], qw[2], qw[1], bias=bias, x_scale=g if fmt == "nvfp4_static" else None,
                                              out_dtype=torch.bfloat16)
        q, s = backend.quantize_nvfp4(x, g)
        ref = backend.scaled_mm_nvfp4(q, qw[0], g, qw[2], s, qw[1], bias=bias, out_dtype=torch.bfloat16)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.nan_to_num(got), torch.nan_to_num(ref))
