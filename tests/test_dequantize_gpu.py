"""GPU parity of the dequantizers: bit-exact against the golden fixtures and the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch
from conftest import golden_names, load_golden
from gpu_util import bits, dit_activation, layout_scale

from oracle import ck_oracle as oc

pytestmark = pytest.mark.gpu
DTYPES = [(torch.float32, "float32", "deq"), (torch.bfloat16, "bfloat16", "deq_bf16"), (torch.float16, "float16", "deq_f16")]


@pytest.fixture(scope="module")
def ck(cuda_device):
    import comfy_kitchen

    assert comfy_kitchen.list_backends()["cuda"]["available"]
    return comfy_kitchen


def _as_bits32(t: torch.Tensor) -> np.ndarray:
    return t.float().cpu().numpy().view(np.uint32)


def _golden_f32(a: np.ndarray, kind: str) -> np.ndarray:
    if kind == "float32":
        return a
    if kind == "bfloat16":
        return oc.bf16_bits_to_f32(a)
    return a.view(np.float16).astype(np.float32)


@pytest.mark.parametrize("name", golden_names("nvfp4_"))
@pytest.mark.parametrize("dtype,kind,key", DTYPES)
def test_nvfp4_golden(ck, cuda_device, name, dtype, kind, key):
    d = load_golden(name)
    q = torch.from_numpy(d["codes"]).to(cuda_device)
    s = torch.from_numpy(d["scales"]).to(cuda_device).view(torch.float8_e4m3fn)
    out = ck.dequantize_nvfp4(q, torch.tensor(float(d["scale"]), device=cuda_device), s, dtype, hi_first=bool(d["hi_first"]))
    assert out.dtype == dtype and tuple(out.shape) == (d["codes"].shape[0], d["codes"].shape[1] * 2)
    np.testing.assert_array_equal(_as_bits32(out), _golden_f32(d[key], kind).view(np.uint32))


@pytest.mark.parametrize("name", golden_names("mxfp8_"))
@pytest.mark.parametrize("dtype,kind,key", DTYPES)
def test_mxfp8_golden(ck, cuda_device, name, dtype, kind, key):
    d = load_golden(name)
    q = torch.from_numpy(d["data"]).to(cuda_device).view(torch.float8_e4m3fn)
    s = torch.from_numpy(d["scales"]).to(cuda_device).view(torch.float8_e8m0fnu)
    out = ck.dequantize_mxfp8(q, s, dtype)
    got, want = _as_bits32(out), _golden_f32(d[key], kind).view(np.uint32)
    finite = np.isfinite(_golden_f32(d[key], kind))  # out-of-domain blocks decode to NaN payloads
    np.testing.assert_array_equal(got[finite], want[finite])


@pytest.mark.parametrize("dtype,kind,key", DTYPES)
def test_round_trip_full_size(ck, cuda_device, dtype, kind, key):
    """[4096,3072] activation: quantize -> dequantize equals the oracle's dequantization, both formats."""
    x = dit_activation(4096, 3072).to(cuda_device)
    sc = layout_scale(x)
    q, s = ck.quantize_nvfp4(x, sc)
    out = ck.dequantize_nvfp4(q, sc, s, dtype)
    ref = oc.dequantize_nvfp4(bits(q), np.float32(sc.item()), bits(s), out_dtype=kind)
    np.testing.assert_array_equal(_as_bits32(out), ref.view(np.uint32))
    q8, s8 = ck.quantize_mxfp8(x)
    out8 = ck.dequantize_mxfp8(q8, s8, dtype)
    ref8 = oc.dequantize_mxfp8(bits(q8), bits(s8), out_dtype=kind)
    np.testing.assert_array_equal(_as_bits32(out8), ref8.view(np.uint32))
    # quantization error bound of the formats: relative error of the round trip
    err = (out.float() - x.float()).norm() / x.float().norm()
    err8 = (out8.float() - x.float()).norm() / x.float().norm()
    assert err < 0.15 and err8 < 0.05


@pytest.mark.parametrize("hi_first", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_nvfp4_two_rows_to_a_thread(cuda_device, dtype, hi_first):
    """From 1185 blocks of one row on (here 1376) a thread of the 16-bit kernels takes two (here the last ones have no second): the
    values of row blocks taken by themselves, which are smaller than that."""
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(11)
    rows, cols, g = 1373, 3088, torch.tensor(0.0123, device=cuda_device)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device)
    q, s = backend.quantize_nvfp4(x, g, hi_first=hi_first)
    got = backend.dequantize_nvfp4(q, g, s, dtype, hi_first=hi_first)
    parts = [backend.dequantize_nvfp4(q[r:r + 128], g, s[r:r + 128], dtype, hi_first=hi_first) for r in range(0, rows, 128)]
    assert rows * cols > 1 << 22 and torch.equal(got, torch.cat(parts))


@pytest.mark.parametrize("rows, cols", [(4736, 1024), (4737, 1024), (4741, 1008)])  # the last size of one row to a thread, the first of two
def test_nvfp4_edge_of_two_rows_to_a_thread(cuda_device, rows, cols):
    from comfy_kitchen.backends import cuda as backend

    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    g = torch.tensor(0.0123, device=cuda_device)
    q, s = backend.quantize_nvfp4(torch.randn(rows, cols, generator=gen, device=cuda_device), g)
    got = backend.dequantize_nvfp4(q, g, s, torch.bfloat16)
    parts = [backend.dequantize_nvfp4(q[r:r + 128], g, s[r:r + 128], torch.bfloat16) for r in range(0, rows, 128)]
    assert torch.equal(got, torch.cat(parts))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows, cols", [(592, 1024), (596, 1024), (3552, 1024), (3556, 1024), (5920, 1024), (5924, 1024)])  # 1, 6, 10 blocks an SM, and more
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_back_to_back_with_a_reader(cuda_device, fmt, rows, cols, dtype):
    """However early a dequantizer lets the next kernel's blocks in, that kernel reads what it wrote: chains on changing data."""
    from comfy_kitchen.backends import cuda as backend

    if fmt == "mxfp8":
        cols *= 2  # the same number of blocks
    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    xs = [torch.randn(rows, cols, generator=gen, device=cuda_device).bfloat16() * s for s in (1, 30, 0.1)]
    if fmt == "mxfp8":
        qs = [backend.quantize_mxfp8(x) for x in xs]
        deq = [lambda q=q: backend.dequantize_mxfp8(*q, dtype) for q in qs]
    else:
        qs = [backend.quantize_nvfp4_dynamic(x) for x in xs]
        deq = [lambda q=q: backend.dequantize_nvfp4(q[0], q[2], q[1], dtype) for q in qs]
    want = []
    for d in deq:
        y = d()
        torch.cuda.synchronize()
        want.append(tuple(t.view(torch.uint8).clone() for t in backend.quantize_mxfp8(y)))
        torch.cuda.synchronize()
    for _ in range(15):
        got = [backend.quantize_mxfp8(d()) for d in deq]
        assert all(torch.equal(g.view(torch.uint8), w) for pair, ref in zip(got, want) for g, w in zip(pair, ref))
