"""Two threads on one stream, inputs of very different magnitudes: the same bits as one after the other."""
from __future__ import annotations

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["from_float", "linear_nvfp4", "linear_mxfp8"])
def test_two_threads_on_one_stream(cuda_device, entry):
    from comfy_kitchen.modules import MXFP8Linear, NVFP4Linear
    from comfy_kitchen.tensor import QuantizedTensor

    gen = torch.Generator(device=cuda_device).manual_seed(5)
    xs = [torch.randn(rows, 512, generator=gen, device=cuda_device, dtype=torch.float32).bfloat16() * s for rows, s in ((96, 1e-2), (700, 1e2))]
    dense = torch.nn.Linear(512, 256, device=cuda_device, dtype=torch.bfloat16)
    if entry == "from_float":
        def call(x):
            q = QuantizedTensor.from_float(x, "TensorCoreNVFP4Layout")
            return q._qdata, q._params.scale, q._params.block_scale.view(torch.uint8)
    else:
        layer = (NVFP4Linear if entry == "linear_nvfp4" else MXFP8Linear).from_linear(dense)

        def call(x):
            return (layer(x),)
    with torch.inference_mode():
        want = [call(x) for x in xs]
    got = [[], []]

    def work(i):
        with torch.inference_mode():
            for _ in range(100):
                got[i].append(call(xs[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        assert len(got[i]) == 100
        for outs in got[i]:
            for a, b in zip(outs, want[i]):
                assert torch.equal(a, b)
