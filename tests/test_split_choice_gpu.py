"""How many CTAs share a tile's K range: enough of the chip is used wherever K is split."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def splits(cuda_device):
    from comfy_kitchen.backends import cuda as backend

    lib = backend.load_library()
    return lambda mx, m, n, k, dtype=2: lib.ck_debug_gemm_splits(int(mx), dtype, m, n, k)


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
    assert splits(mx, 4096, 3072, 12288) == 1   # many tiles
    assert splits(mx, 0, 128, 4096) < 0
