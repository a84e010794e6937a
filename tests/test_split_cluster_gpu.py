"""Split-K GEMMs whose partial tiles a thread-block cluster adds through distributed shared memory:
every cluster size, ragged rows / columns / K, all result types, and the entry points that reach it."""
from __future__ import annotations

import pytest
import torch
from gpu_util import layout_scale
from test_gemm_gpu import _check_mxfp8, _check_nvfp4, _operands, ck, gemm_status  # noqa: F401  (ck is a fixture)

pytestmark = pytest.mark.gpu

# few rows (operands swapped): 1 .. 32 rows, N not a multiple of 128, K with a short last stage;
# 128 x 128 tiles: one row past the swapped path, partial row / column tiles
SHAPES = [(1, 128, 4096), (32, 136, 4640), (17, 6272, 8192), (5, 520, 12320),
          (33, 128, 4096), (129, 264, 12320), (300, 1032, 8192), (64, 2312, 6176), (512, 1160, 4128)]


def _splits(mx: bool, m: int, n: int, k: int) -> int:
    from comfy_kitchen.backends import cuda as backend

    return backend.load_library().ck_debug_gemm_splits(int(mx), 2, m, n, k, 1)


@pytest.mark.parametrize("shape", SHAPES)
def test_split_cluster_against_oracle(ck, cuda_device, shape):  # noqa: F811
    m, n, k = shape
    assert _splits(True, m, n, k) > 1  # and NVFP4 from twice MXFP8's 18 stages (16 up to 32 rows) on
    assert (_splits(False, m, n, k) > 1) == (k >= (4096 if m <= 32 else 17 * 256 + 1))
    a, b, bias = _operands(m, n, k, seed=3 * m + n + k)
    for dtype, with_bias in ((torch.float32, bias), (torch.bfloat16, None), (torch.float16, bias)):
        _check_nvfp4(ck, cuda_device, a, b, with_bias, dtype)
        _check_mxfp8(ck, cuda_device, a, b, with_bias, dtype)
    assert gemm_status() == 0


# up to 8 rows on 8 CTAs a quarter tile per warp, beyond whole tiles of a row, beyond 32 rows the plain tiles; the last
# three go through a workspace
@pytest.mark.parametrize("shape", [(7, 264, 8192), (8, 264, 8192), (20, 264, 8192), (32, 6144, 12288), (130, 264, 8192),
                                   (250, 3000, 12288), (256, 3072, 6144), (129, 2184, 16384)])
def test_split_cluster_against_the_unsplit_tiles(ck, cuda_device, shape, monkeypatch):  # noqa: F811
    """fp32 results: only the order of the fp32 sums differs (at most 8 partial sums of one K range
    each: 2^-24 per addition, relative to the sums' magnitudes; 1e-5 leaves a factor of 20).  A result
    that does not start on 16 bytes is stored value by value up to 32 rows and takes the unsplit tiles
    beyond."""
    from comfy_kitchen.backends import cuda as backend

    m, n, k = shape
    assert _splits(False, m, n, k) > 1
    a, b, _ = _operands(m, n, k, seed=m + n)
    sa, sb = layout_scale(a).to(cuda_device), layout_scale(b).to(cuda_device)
    qa, bsa = ck.quantize_nvfp4(a.to(cuda_device), sa)
    qb, bsb = ck.quantize_nvfp4(b.to(cuda_device), sb)
    got = ck.scaled_mm_nvfp4(qa, qb, sa, sb, bsa, bsb, out_dtype=torch.float32)
    monkeypatch.setenv("CK_GEMM_CONFIG", "1")
    ref = ck.scaled_mm_nvfp4(qa, qb, sa, sb, bsa, bsb, out_dtype=torch.float32)
    monkeypatch.delenv("CK_GEMM_CONFIG")
    assert ((got - ref).norm() / ref.norm()).item() <= 1e-5
    lib = backend.load_library()
    room = torch.empty(m * n + 1, device=cuda_device)
    off = room[1:]
    assert lib.ck_scaled_mm_nvfp4(qa.data_ptr(), qb.data_ptr(), bsa.data_ptr(), bsb.data_ptr(), sa.data_ptr(), sb.data_ptr(), None,
                                  None, 0, off.data_ptr(), 0, m, n, k, torch.cuda.current_stream().cuda_stream) == 0
    assert ((off.view(m, n) - ref).norm() / ref.norm()).item() <= 1e-5
    assert gemm_status() == 0


@pytest.mark.parametrize("shape", [(1, 1024, 8192), (256, 640, 8192)])
def test_one_call_linear_takes_the_same_split(ck, cuda_device, shape):  # noqa: F811
    from comfy_kitchen.backends import cuda as backend

    m, n, k = shape
    a, b, bias = _operands(m, n, k, seed=m)
    x, bias = a.to(cuda_device), bias.to(cuda_device)
    qb, bsb = ck.quantize_mxfp8(b.to(cuda_device))
    qa, bsa = ck.quantize_mxfp8(x)
    y = backend.linear_mxfp8_from_float(x, qb, bsb, bias=bias, out_dtype=torch.bfloat16)
    assert torch.equal(y, ck.scaled_mm_mxfp8(qa, qb, bsa, bsb, bias=bias, out_dtype=torch.bfloat16))
