"""How many CTAs share a tile's K range: enough of the chip is used wherever K is split."""
from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def splits(cuda_device):
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    return lambda mx, m, n, k, dtype=2, workspace=0: lib.ck_debug_gemm_splits(int(mx), dtype, m, n, k, workspace)


@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("mx", [False, True])
@pytest.mark.parametrize("rows", [5, 16, 32])
@pytest.mark.parametrize("n", [128, 2048, 3072, 4096, 5120, 6144, 6272])
def test_few_rows(splits, cuda_device, n, rows, mx, dtype):
    """Up to 32 rows, from 24 pipeline stages on (256 elements of NVFP4, 128 of MXFP8): at most ten stages a CTA, or
    more CTAs than SMs (a cluster of one more finds no room: 32 tiles of six are 192 on 148)."""
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    for stages in (24, 48, 96):
        s = splits(mx, rows, n, stages * (128 if mx else 256), dtype)
        assert 2 <= s <= 8
        tiles = -(-n // 128)
        assert -(-stages // s) <= 10 or s == 8 or s * tiles > 1.25 * sms, (stages, s)


@pytest.mark.parametrize("mx", [False, True])
def test_not_split(splits, mx):
    assert splits(mx, 1, 6400, 12288) == 1      # more than a third of the SMs have a tile
    assert splits(mx, 32, 1024, 1024) == 1      # a short K
    assert splits(mx, 128, 3072, 17 * (128 if mx else 256)) == 1  # tiles of which two CTAs would come
    assert splits(mx, 128, 3072, 18 * (128 if mx else 256)) == 3
    assert splits(mx, 4096, 3072, 12288) == 1   # many tiles
    assert splits(mx, 0, 128, 4096) < 0


@pytest.mark.parametrize("mx", [False, True])
@pytest.mark.parametrize("m, n, stages", [(256, 3072, 24), (256, 3072, 48), (128, 6272, 96), (250, 3000, 32), (256, 2304, 64)])
def test_workspace_takes_the_split_that_clusters_cannot(splits, cuda_device, mx, m, n, stages):
    """Tiles whose clusters leave SMs idle (148 SMs in parts of about 16 to 20: 45 clusters of three, 33 of four)."""
    from comfy_kitchen.backends import cuda as backend

    k = stages * (128 if mx else 256)
    tiles = -(-m // 128) * -(-n // 128)
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    assert splits(mx, m, n, k) < splits(mx, m, n, k, workspace=1) == sms // tiles
    assert backend.load_library().ck_scaled_mm_workspace_bytes(int(mx), m, n, k) == (sms // tiles) * m * n * 4


@pytest.mark.parametrize("mx", [False, True])
@pytest.mark.parametrize("m, n, stages", [(256, 2304, 48), (128, 2304, 96), (128, 1024, 96), (256, 3072, 16), (32, 6144, 96)])
def test_on_chip(splits, mx, m, n, stages):
    from comfy_kitchen.backends import cuda as backend

    k = stages * (128 if mx else 256)
    assert splits(mx, m, n, k) == splits(mx, m, n, k, workspace=1)
    assert backend.load_library().ck_scaled_mm_workspace_bytes(int(mx), m, n, k) == 256


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_workspace_and_clusters_agree(cuda_device, fmt, dtype):
    """The same sums of one K range each, added in split order, over two or three ranges: 2^-24 per addition, relative
    to the sums' magnitudes (1e-5 leaves a factor of 20), and the result type's rounding (2^-8 for bf16, half of it
    from either side)."""
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    m, n, k = 250, 3000, 8192
    mx = fmt == "mxfp8"
    gen = torch.Generator(device=cuda_device).manual_seed(9)
    a, b = (torch.randn(r, k, generator=gen, device=cuda_device) for r in (m, n))
    one, bias = torch.tensor(0.01, device=cuda_device), torch.linspace(-9, 9, n, device=cuda_device)
    (qa, sa), (qb, sb) = ((backend.quantize_mxfp8(t) if mx else backend.quantize_nvfp4(t, one)) for t in (a, b))
    need = lib.ck_scaled_mm_workspace_bytes(int(mx), m, n, k)
    assert need > 256
    code = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype]
    outs = {}
    for name, nbytes in (("null", None), ("short", need - 1), ("full", need)):
        ws = None if nbytes is None else torch.full((nbytes,), 0xFF, dtype=torch.uint8, device=cuda_device)  # NaNs
        out = torch.full((m, n), float("nan"), dtype=dtype, device=cuda_device)
        scales = () if mx else (one.data_ptr(), one.data_ptr(), None)
        call = lib.ck_scaled_mm_mxfp8_ws if mx else lib.ck_scaled_mm_nvfp4_ws
        rc = call(qa.data_ptr(), qb.data_ptr(), sa.data_ptr(), sb.data_ptr(), *scales, bias.data_ptr(), 0, out.data_ptr(), code, m, n, k,
                  None if ws is None else ws.data_ptr(), nbytes or 0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.ck_last_error()
        outs[name] = out
    assert torch.equal(outs["null"], outs["short"])
    ref = outs["null"].float()
    bound = {torch.float32: 1e-5, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[dtype]
    assert ((outs["full"].float() - ref).norm() / ref.norm()).item() <= bound
    status = ctypes.c_int(-1)
    assert lib.ck_gemm_status(ctypes.byref(status)) == 0 and status.value == 0


# (rows, columns, stages) of every number of CTAs per tile, operands swapped (up to 32 rows) and not
@pytest.mark.parametrize("m, n, stages, want", [
    (9, 6144, 16, 2), (1, 5120, 16, 3), (32, 128, 16, 4), (3, 128, 20, 5), (31, 136, 24, 6), (1, 128, 28, 7), (17, 1024, 32, 8),
    (40, 8192, 24, 2), (33, 128, 18, 3), (130, 264, 25, 4), (257, 128, 30, 5), (64, 520, 36, 6), (128, 128, 42, 7), (129, 384, 48, 8)])
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
def test_every_cluster_size(splits, cuda_device, monkeypatch, fmt, m, n, stages, want):
    """Against the unsplit 128 x 128 tiles; the bound as in test_workspace_and_clusters_agree."""
    from comfy_kitchen.backends import cuda as backend

    mx = fmt == "mxfp8"
    k = stages * (128 if mx else 256) - 32  # a short last stage
    assert splits(mx, m, n, k, dtype=0) == want == splits(mx, m, n, k, dtype=0, workspace=1)
    gen = torch.Generator(device=cuda_device).manual_seed(stages)
    a, b = (torch.randn(r, k, generator=gen, device=cuda_device) for r in (m, n))
    one, bias = torch.tensor(0.01, device=cuda_device), torch.linspace(-9, 9, n, device=cuda_device)
    if mx:
        (qa, sa), (qb, sb) = backend.quantize_mxfp8(a), backend.quantize_mxfp8(b)

        def call():
            return backend.scaled_mm_mxfp8(qa, qb, sa, sb, bias=bias, out_dtype=torch.float32)
    else:
        (qa, sa), (qb, sb) = backend.quantize_nvfp4(a, one), backend.quantize_nvfp4(b, one)

        def call():
            return backend.scaled_mm_nvfp4(qa, qb, one, one, sa, sb, bias=bias, out_dtype=torch.float32)
    got = call()
    monkeypatch.setenv("CK_GEMM_CONFIG", "1")
    ref = call()
    monkeypatch.delenv("CK_GEMM_CONFIG")
    assert ((got - ref).norm() / ref.norm()).item() <= 1e-5
