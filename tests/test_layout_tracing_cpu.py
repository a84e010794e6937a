"""The layouts quantize tensors whose sizes are symbolic: the operators are recorded, with the padding decided by guards, and nothing
asks for a number that there is not."""
from __future__ import annotations

import pytest
import torch
from torch.fx.experimental.proxy_tensor import make_fx

from comfy_kitchen.tensor import QuantizedTensor


@pytest.fixture(scope="module", autouse=True)
def loaded():
    """As in a program that has called the backend before: with the library and the native half."""
    from comfy_kitchen.backends import cuda as backend

    try:
        backend.load_library()
    except RuntimeError as e:
        pytest.skip(str(e))


@pytest.mark.parametrize("transform", [lambda f: f, torch.func.functionalize])  # the latter's tensors are of the plain type
@pytest.mark.parametrize("shape", [(64, 128), (33, 70), (2048, 96)])  # no padding, both sides padded, more than 128 KiB
@pytest.mark.parametrize("layout, op, static", [("TensorCoreNVFP4Layout", "quantize_nvfp4", False), ("TensorCoreNVFP4Layout", "quantize_nvfp4", True),
                                                ("TensorCoreMXFP8Layout", "quantize_mxfp8", False)])
def test_symbolic_shapes(layout, op, static, shape, transform):
    def quantize(x, scale):
        q = QuantizedTensor.from_float(x, layout, **({"scale": scale} if static else {}))
        return q._qdata, q._params.scale

    graph = make_fx(transform(quantize), tracing_mode="symbolic")(torch.randn(shape), torch.tensor(0.1)).graph
    recorded = [node for node in graph.nodes if node.target is getattr(torch.ops.comfy_kitchen, op).default]
    granule = 32 if op == "quantize_mxfp8" else 16
    assert len(recorded) == 1 and recorded[0].args[-2 if granule == 16 else -1] is any(n % granule for n in shape)
