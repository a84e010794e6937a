"""The native half of the wrappers: the bits of the Python wrappers, and None (the wrapper's own way) for every call
that is not a plain eager one."""
from __future__ import annotations

import threading
import timeit

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import comfy_kitchen as ck
from comfy_kitchen.ops import host_operator

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend(cuda_device):
    from comfy_kitchen.backends import cuda as backend

    assert backend._host is not None, "lib/_ck_host.so is not built or does not load"
    return backend


def _calls(backend, device, rows, dtype):
    gen = torch.Generator(device=device).manual_seed(rows)
    x = torch.randn(rows, 256, generator=gen, device=device).to(dtype)
    w = torch.randn(128, 256, generator=gen, device=device).bfloat16()
    g, bias = torch.tensor(0.01, device=device), torch.linspace(-1, 1, 128, device=device)
    q4, q8 = backend.quantize_nvfp4(w, g), backend.quantize_mxfp8(w)
    x4, x8 = backend.quantize_nvfp4(x, g), backend.quantize_mxfp8(x)
    return {
        "quantize_nvfp4": (x, g), "quantize_nvfp4_dynamic": (x, True), "quantize_mxfp8": (x, True),
        "dequantize_nvfp4": (q4[0], g, q4[1], dtype), "dequantize_mxfp8": (*q8, dtype),
        "scaled_mm_nvfp4": (x4[0], q4[0], g, g, x4[1], q4[1], bias, dtype),
        "scaled_mm_mxfp8": (x8[0], q8[0], x8[1], q8[1], None, None),
        "linear_nvfp4_from_float": (x, q4[0], g, q4[1], None, None, None),
        "linear_mxfp8_from_float": (x, *q8, bias, torch.float16),
    }


def _equal(a, b):
    a, b = ((t,) if isinstance(t, torch.Tensor) else t for t in (a, b))
    assert len(a) == len(b)
    for u, v in zip(a, b):
        assert type(u) is type(v) is torch.Tensor and u.dtype == v.dtype and u.shape == v.shape and u.stride() == v.stride()
        assert u.is_inference() == v.is_inference() and torch.equal(u.view(torch.uint8) if u.dim() else u, v.view(torch.uint8) if v.dim() else v)


@pytest.mark.parametrize("inference", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [1, 40, 300])
def test_same_as_the_python_wrappers(backend, cuda_device, monkeypatch, rows, dtype, inference):
    with torch.inference_mode(inference):
        calls = _calls(backend, cuda_device, rows, dtype)
        got = {name: getattr(backend, name)(*args) for name, args in calls.items()}
        monkeypatch.setattr(backend, "_host", None)
        for name, args in calls.items():
            _equal(got[name], getattr(backend, name)(*args))
    backend.check_device_status("host half")


def test_none_for_calls_that_are_not_plain(backend, cuda_device, monkeypatch):
    host = backend._host
    x, g = torch.randn(32, 64, device=cuda_device), torch.tensor(0.01, device=cuda_device)

    def plain(x=x, g=g, pad=False, hi=True):
        return host.quantize_nvfp4(x, g, pad, hi) is not None

    assert plain() and plain(torch.nn.Parameter(x, requires_grad=False))
    assert not plain(x.cpu()) and not plain(x.double()) and not plain(x.t()) and not plain(x[0]) and not plain(x[:0]) and not plain(pad=1)
    assert not plain(g=g.double()) and not plain(g=g.cpu()) and not plain(g=0.01) and not plain(g=torch.ones(2, device=cuda_device)) and not plain("x")
    assert not plain(torch._neg_view(x))
    assert not plain(x[:, :40].contiguous()) and plain(x[:, :40].contiguous(), pad=True)  # 40 columns are no whole blocks
    leaf = x.clone().requires_grad_()
    assert not plain(leaf)
    with torch.no_grad():
        assert plain(leaf)

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert not plain()
    with torch.overrides.TorchFunctionMode():
        assert not plain()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert not plain()
    torch.func.vmap(lambda t: (t, plain() and pytest.fail("functorch is active"))[0])(x)
    with monkeypatch.context() as m:
        m.setenv("CK_STRICT", "1")
        assert not plain()
    with torch.autocast("cuda"):
        assert plain()
    assert plain()


def test_refusing_costs_no_exception(backend, cuda_device):
    """A call that is refused late goes to the Python wrapper all the same: asking costs less than a view of a tensor does (0.2 to
    0.3 us against 0.6; 1.3 to 1.7 with a C++ exception)."""
    host = backend._host
    x, g, bias = torch.randn(32, 64, device=cuda_device), torch.tensor(0.01, device=cuda_device), torch.zeros(9, device=cuda_device)
    codes, scales = backend.quantize_nvfp4(x, g)
    leaf, cube, t, shifted = x.clone().requires_grad_(), x.view(2, 16, 64), x.t(), torch.zeros(32 * 64 + 1, device=cuda_device)[1:].view(32, 64)
    refused = [lambda: host.quantize_nvfp4(leaf, g, False, True), lambda: host.quantize_mxfp8(t, False), lambda: host.quantize_mxfp8(cube, False),
               lambda: host.linear_nvfp4_from_float(shifted, codes, g, scales, None, None, None),
               lambda: host.linear_nvfp4_from_float(x, codes, g, scales, bias, None, None)]

    def cost(call):
        return min(timeit.repeat(call, number=200, repeat=20)) / 200

    view = cost(x.t)
    for call in refused:
        assert call() is None and cost(call) < 1.5 * view


def test_operators_ask_the_registry(backend, cuda_device, monkeypatch):
    assert host_operator("quantize_nvfp4") is not None
    ck.disable_backend("cuda")
    try:
        assert host_operator("quantize_nvfp4") is None
    finally:
        ck.enable_backend("cuda")
    with ck.use_backend("cuda"):
        assert host_operator("quantize_nvfp4") is None
    with torch.autograd.forward_ad.dual_level():
        assert host_operator("quantize_nvfp4") is None
    with monkeypatch.context() as m:
        m.setattr(backend, "quantize_nvfp4", lambda **kw: "somebody's own")
        assert ck.quantize_nvfp4(torch.randn(32, 64, device=cuda_device), torch.tensor(0.01, device=cuda_device)) == "somebody's own"
    assert host_operator("quantize_nvfp4") is not None


def test_side_streams_and_threads(backend, cuda_device):
    """Results and workspaces belong to the current stream of the calling thread."""
    from comfy_kitchen.modules import MXFP8Linear, NVFP4Linear

    dense = torch.nn.Linear(512, 256, device=cuda_device, dtype=torch.bfloat16)
    layers = [NVFP4Linear.from_linear(dense), MXFP8Linear.from_linear(dense)]
    gen = torch.Generator(device=cuda_device).manual_seed(4)
    xs = [torch.randn(r, 512, generator=gen, device=cuda_device).bfloat16() * s for r, s in ((700, 1e-2), (96, 1e2), (5, 1.0))]
    with torch.inference_mode():
        want = [[layer(x) for layer in layers] for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        with torch.inference_mode(), torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(60):
                for layer, ref in zip(layers, want[i]):
                    if not torch.equal(layer(xs[i]), ref):
                        bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
