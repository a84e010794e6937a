"""The streaming quantizer: dynamic scale finished inside it, fp32 inputs, padded rows - against the
one-kernel scale and the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch
from gpu_util import as_f32, bits

from oracle import ck_oracle as oc

pytestmark = pytest.mark.gpu

# inputs that every block reads whole (up to 64 KiB with at most eight rows, else 128 KiB) and larger ones;
# more partial maxima than threads of a block; one unit; a column chunk of one unit; rows of padding
# only in the last group; columns that take the general kernel (16, 48: 16-bit types; 65: padded)
SHAPES = [(1, 32), (16, 1024), (32, 1024), (33, 1024), (3, 2080), (130, 96), (1003, 3072), (2500, 4096), (40, 48), (7, 16), (33, 65)]


@pytest.fixture(scope="module")
def backend(cuda_device):
    from comfy_kitchen.backends import cuda as backend

    backend.load_library()
    return backend


def _input(m, k, dtype):
    g = torch.Generator(device="cpu").manual_seed(m * 7 + k)
    x = torch.randn(m, k, generator=g)
    x[:, : max(1, k // 5)] *= 1e-3
    x[m // 2] = 0.0
    x[-1, -1] = -37.5  # the maximum: last element of the input
    return x.to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", SHAPES)
def test_dynamic_scale_in_the_quantizer(backend, cuda_device, shape, dtype):
    m, k = shape
    x = _input(m, k, dtype)
    pad = m % 16 != 0 or k % 16 != 0
    dev = x.to(cuda_device)
    for hi_first in (True, False):
        codes, block_scales, scale = backend.quantize_nvfp4_dynamic(dev, pad_16x=pad, hi_first=hi_first)
        want = backend.nvfp4_tensor_scale(dev)
        assert scale.view(torch.int32).item() == want.view(torch.int32).item()
        padded = torch.nn.functional.pad(x, (0, -k % 16, 0, -m % 16)) if pad else x
        ref_codes, ref_scales = oc.quantize_nvfp4(as_f32(padded), np.float32(scale.item()), hi_first=hi_first)
        assert np.array_equal(bits(codes), ref_codes)
        assert np.array_equal(bits(block_scales), ref_scales)
        static_codes, static_scales = backend.quantize_nvfp4(dev, scale, pad_16x=pad, hi_first=hi_first)
        assert torch.equal(static_codes, codes) and torch.equal(static_scales.view(torch.uint8), block_scales.view(torch.uint8))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_dynamic_quantizer_leaves_a_shared_scratch_usable(backend, cuda_device, dtype):
    """The first word of the scratch is the arrival counter of the one-kernel scale, which may use the
    same scratch in between; an input that starts off a 32-byte boundary takes the general kernel."""
    lib = backend.load_library()
    code = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype]
    x = _input(300, 1056, dtype).to(cuda_device)
    off = torch.empty(300 * 1056 + 1, dtype=dtype, device=cuda_device)[1:].view(300, 1056)
    off.copy_(x)
    need = lib.ck_quantize_nvfp4_dynamic_scratch_bytes(x.numel())
    scratch = torch.zeros(need, dtype=torch.uint8, device=cuda_device)
    codes, scales, scale = backend.quantize_nvfp4_dynamic(x, pad_16x=False)
    stream = torch.cuda.current_stream().cuda_stream
    for src in (x, off, x):
        out, one = torch.empty((), device=cuda_device), torch.empty((), device=cuda_device)
        q, s = torch.empty_like(codes), torch.empty_like(scales)
        assert lib.ck_quantize_nvfp4_dynamic(src.data_ptr(), code, out.data_ptr(), q.data_ptr(), s.data_ptr(), 300, 1056, 300, 1056, 1,
                                             scratch.data_ptr(), need, stream) == 0, lib.ck_last_error()
        assert lib.ck_nvfp4_tensor_scale(src.data_ptr(), code, src.numel(), one.data_ptr(), scratch.data_ptr(), need, stream) == 0
        assert torch.equal(out, scale) and torch.equal(one, scale)
        assert torch.equal(q, codes) and torch.equal(s.view(torch.uint8), scales.view(torch.uint8))
    assert lib.ck_quantize_nvfp4_dynamic(x.data_ptr(), code, out.data_ptr(), q.data_ptr(), s.data_ptr(), 300, 1056, 300, 1056, 1,
                                         scratch.data_ptr(), need - 1, stream) != 0
    assert f"scratch of {need - 1} bytes, {need} needed".encode() in lib.ck_last_error()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [1, 8, 9, 128])
def test_inputs_that_are_read_whole_leave_the_scratch_alone(backend, cuda_device, monkeypatch, rows, dtype):
    """On both sides of the line that the library reports: nothing is written to the scratch up to it; beyond it there are partial
    maxima.  What the wrappers keep and share is asked for on this side of the lowest line alone, by them and by the layout."""
    from comfy_kitchen.tensor import QuantizedTensor

    asked, kept = [], backend.kept_scratch
    monkeypatch.setattr(backend, "kept_scratch", lambda t: asked.append(t.shape) or kept(t))
    lib = backend.load_library()
    code, elem = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype], torch.empty((), dtype=dtype).element_size()
    line = lib.ck_quantize_nvfp4_dynamic_whole_input_bytes(rows) // elem // rows // 32 * 32
    for k in (line, line + 32):
        x = _input(rows, k, dtype).to(cuda_device)
        need = lib.ck_quantize_nvfp4_dynamic_scratch_bytes(x.numel())
        scratch = torch.full((need,), 0xA5, dtype=torch.uint8, device=cuda_device)
        want = backend.quantize_nvfp4_dynamic(x, pad_16x=False)
        out, q, s = torch.empty((), device=cuda_device), torch.empty_like(want[0]), torch.empty_like(want[1])
        assert lib.ck_quantize_nvfp4_dynamic(x.data_ptr(), code, out.data_ptr(), q.data_ptr(), s.data_ptr(), rows, k, rows, k, 1,
                                             scratch.data_ptr(), need, torch.cuda.current_stream().cuda_stream) == 0, lib.ck_last_error()
        assert bool((scratch == 0xA5).all()) == (k == line)
        assert torch.equal(out, want[2]) and torch.equal(q, want[0]) and torch.equal(s.view(torch.uint8), want[1].view(torch.uint8))
        QuantizedTensor.from_float(x, "TensorCoreNVFP4Layout")
        assert asked == [x.shape] * (2 if x.nbytes <= lib.ck_quantize_nvfp4_dynamic_whole_input_bytes(1) else 0)
        asked.clear()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(1003, 3072), (1, 32), (129, 96), (31, 2080)])
def test_mxfp8_padded_rows(backend, cuda_device, shape, dtype):
    m, k = shape
    x = _input(m, k, dtype)
    data, scales = backend.quantize_mxfp8(x.to(cuda_device), pad_32x=True)
    ref, ref_scales = oc.quantize_mxfp8(as_f32(torch.nn.functional.pad(x, (0, 0, 0, -m % 32))))
    assert np.array_equal(bits(data), ref.view(np.uint8)) and np.array_equal(bits(scales), ref_scales.view(np.uint8))
