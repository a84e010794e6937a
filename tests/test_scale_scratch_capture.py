"""The tensor-scale kernel's scratch starts at zero and is kept between calls: not the one of a captured call, whose zeros are written
when its graph runs, if it ever does."""
from __future__ import annotations

import pytest
import torch

from comfy_kitchen.backends import cuda as backend


def test_a_captured_call_keeps_none(monkeypatch):
    cpu = torch.device("cpu")
    monkeypatch.setattr(backend, "_scale_scratch", {})
    monkeypatch.setattr(backend, "_capturing", lambda: True)
    first, second = backend._scale_scratch_for(cpu, 5, 300), backend._scale_scratch_for(cpu, 5, 300)
    assert first.data_ptr() != second.data_ptr() and not first.any() and min(first.numel(), second.numel()) >= 300
    assert not backend._scale_scratch
    monkeypatch.setattr(backend, "_capturing", lambda: False)
    kept = backend._scale_scratch_for(cpu, 5, 300)
    monkeypatch.setattr(backend, "_capturing", lambda: True)
    assert backend._scale_scratch_for(cpu, 5, 300) is kept  # zeroed by a call that ran
    assert backend._scale_scratch_for(cpu, 5, kept.numel() + 1) is not kept and backend._scale_scratch_for(cpu, 5, 300) is kept


@pytest.mark.gpu
@pytest.mark.parametrize("rows, cols", [(8, 64), (70, 40)])  # inside the quantizer; the one-kernel scale (padded columns)
def test_graphs_of_a_stream_that_ran_nothing_before(cuda_device, rows, cols):
    """The second graph's result does not hang on the first one having run."""
    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    x = torch.randn(rows, cols, generator=gen, device=cuda_device).bfloat16()
    want = [t.clone() for t in backend.quantize_nvfp4_dynamic(x, True)]
    side, graphs, got = torch.cuda.Stream(), [], []
    for _ in range(2):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=side):
            got.append(backend.quantize_nvfp4_dynamic(x, True))
    assert (cuda_device, side.cuda_stream) not in backend._scale_scratch
    for i in (1, 0, 1):
        for t in got[i]:
            t.view(torch.uint8).fill_(0xFF) if t.dim() else t.fill_(float("nan"))
        graphs[i].replay()
        assert all(torch.equal(a.view(torch.uint8) if a.dim() else a, b.view(torch.uint8) if b.dim() else b) for a, b in zip(got[i], want))
