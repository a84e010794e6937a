"""Two threads on one stream, and two graphs captured on one stream that replay side by side, with inputs of very
different magnitudes: the same bits as one after the other."""
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


@pytest.mark.parametrize("entry", ["from_float", "linear_nvfp4", "linear_mxfp8", "scaled_mm"])
def test_graphs_captured_on_one_stream(cuda_device, entry):
    """A captured call has a workspace of its own, whatever the capturing thread had on that stream before."""
    import comfy_kitchen as ck
    from comfy_kitchen.modules import MXFP8Linear, NVFP4Linear
    from comfy_kitchen.tensor import QuantizedTensor

    gen = torch.Generator(device=cuda_device).manual_seed(6)
    k = 8192 if entry == "scaled_mm" else 512
    xs = [torch.randn(256, k, generator=gen, device=cuda_device, dtype=torch.float32).bfloat16() * s for s in (1e-2, 1e2)]
    if entry == "from_float":
        def call(x):
            q = QuantizedTensor.from_float(x, "TensorCoreNVFP4Layout")
            return q._qdata, q._params.scale
    elif entry == "scaled_mm":  # 256 x 3072: partial tiles through a workspace
        one = torch.tensor(0.01, device=cuda_device)
        w, sw = ck.quantize_nvfp4(torch.randn(3072, k, generator=gen, device=cuda_device), one)
        qs = {x.data_ptr(): ck.quantize_nvfp4(x, one) for x in xs}

        def call(x):
            return (ck.scaled_mm_nvfp4(qs[x.data_ptr()][0], w, one, one, qs[x.data_ptr()][1], sw),)
    else:
        dense = torch.nn.Linear(k, 256, device=cuda_device, dtype=torch.bfloat16)
        layer = (NVFP4Linear if entry == "linear_nvfp4" else MXFP8Linear).from_linear(dense)

        def call(x):
            return (layer(x),)
    with torch.inference_mode():
        want = [call(x) for x in xs]
        capture, sides = torch.cuda.Stream(), [torch.cuda.Stream() for _ in xs]
        graphs, outs = [], []
        with torch.cuda.stream(capture):
            call(xs[0])
        torch.cuda.synchronize()
        for x in xs:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=capture):
                outs.append([call(x) for _ in range(8)])
            graphs.append(graph)
        for _ in range(20):
            for graph, side in zip(graphs, sides):
                with torch.cuda.stream(side):
                    graph.replay()
        torch.cuda.synchronize()
    for i in range(2):
        for out in outs[i]:
            for a, b in zip(out, want[i]):
                assert torch.equal(a, b)
