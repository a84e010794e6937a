"""torch.library custom operators of the quantized-linear path.

Operator names, schemas (dtype passed as an integer code; ``float epsilon, bool
pad_16x, bool hi_first``) and fake (meta) shape functions match the reference's
comfy_kitchen/backends/eager/quantization.py:471-730, so graphs traced against the
reference resolve against this build.  Each operator looks its implementation up in
the registry with keyword arguments, exactly as the reference does (:492-496).
"""
from __future__ import annotations

import torch

from .float_utils import roundup
from .registry import registry

# dtype codes shared with the C ABI (comfy_kitchen/backends/eager/quantization.py:31-39)
DTYPE_CODE_TO_DTYPE = {
    0: torch.float32,
    1: torch.float16,
    2: torch.bfloat16,
    5: torch.float8_e4m3fn,
    6: torch.float8_e5m2,
}
DTYPE_TO_CODE = {v: k for k, v in DTYPE_CODE_TO_DTYPE.items()}


_PLAIN_TYPES = (torch.Tensor, torch.nn.Parameter)
_MAY_BE_PENDING = (torch.float32, torch.bfloat16, torch.float16)  # parts of complex tensors, tangents: no codes or block scales


def _impl(name: str, kwargs: dict):
    return registry.get_implementation(name, kwargs=kwargs)(**kwargs)


# What Python code can register in front of the kernels below, for tensors that need no gradient.
_KEYS_IN_FRONT = ("CUDA", "AutocastCUDA", "AutogradCUDA", "ADInplaceOrView", "BackendSelect")
_registrations = getattr(torch.library, "_impls", None)  # "namespace/operator/key" of every kernel registered from Python
_own: dict = {}  # operator -> (its definition, the kernels it was defined with, the registrations that would precede them)


def _remember(op) -> None:
    name = op._name
    _own[name] = (op, dict(op._backend_fns), frozenset(f"comfy_kitchen/{name}/{key}" for key in _KEYS_IN_FRONT))


def replaced(name: str) -> bool:
    """True when somebody has registered a kernel of their own for the operator (``torch.library.impl``,
    ``register_kernel``, ``register_autocast``) or switched this one off: the dispatcher finds it.  A kernel
    registered from C++ code leaves no trace that is cheap to see; calls through ``torch.ops`` find it."""
    known = _own.get(name)
    if known is None or _registrations is None:
        return True
    op, kernels, in_front = known
    return not in_front.isdisjoint(_registrations) or op._backend_fns != kernels or bool(op._disabled_kernel)


def host_operator(name: str):
    """The operator's implementation as one native function (plain eager calls; None for every other call), or None
    when the dispatcher or the registry has something to decide: a kernel of somebody's own, tracing, forward-mode
    autograd, another backend.  (What the function asks for itself: plain CUDA tensors, no autograd graph, no
    modes, transforms, profilers or observers.)  256 pre-quantized rows took 28 us of host time through the checks of
    :func:`dispatcher_adds_nothing`, the registry and the Python wrapper."""
    if torch.compiler.is_compiling() or replaced(name) or torch.autograd.forward_ad._current_level >= 0:
        return None
    global _cuda_backend
    if _cuda_backend is None:
        from .backends import cuda as _cuda_backend  # imports this module
    return _cuda_backend.host_operator(name)


_cuda_backend = None


def dispatcher_adds_nothing(tensors, optional=()) -> bool:
    """True when calling an operator that nobody replaced (:func:`replaced`) through the torch dispatcher
    would only call its implementation: plain CUDA tensors of no autograd graph, without a pending negation
    or zero, and nobody who watches or rewrites operator calls (tracing, ``torch.compile``, a profiler, a
    torch function or dispatch mode, functorch, forward-mode autograd).  An observer without a profiler
    (``ExecutionTraceObserver`` on its own) cannot be asked for: it sees the call's allocations and not the
    operator's name.

    The call then goes to the registry at once.  The custom-op layer (schema, autograd and view
    wrappers, output alias checks) costs more host time than a GEMM of a few hundred rows takes on the
    device: with it and the wrappers' other overhead gone, 256 pre-quantized rows take 27.9 us instead of
    46.9 through ``scaled_mm_nvfp4``, and dequantizing 12288 x 3072 takes 21.3 instead of 37.8.
    Everything else keeps the dispatcher's route and its errors.
    """
    if torch.compiler.is_compiling() or torch.autograd._profiler_enabled() or torch._C._get_tracing_state() is not None or \
            torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack() or \
            torch._C._functorch.peek_interpreter_stack() is not None or torch.autograd.forward_ad._current_level >= 0:
        return False
    grad = torch.is_grad_enabled()
    for t in tensors:
        if type(t) not in _PLAIN_TYPES or not t.is_cuda or (grad and t.requires_grad):
            return False
        if t.dtype in _MAY_BE_PENDING and (t.is_neg() or t._is_zerotensor()):
            return False
    for t in optional:
        if t is not None and (type(t) not in _PLAIN_TYPES or not t.is_cuda or (grad and t.requires_grad) or t.is_neg() or
                              t._is_zerotensor()):
            return False
    return True


@torch.library.custom_op("comfy_kitchen::quantize_nvfp4", mutates_args=())
def _op_quantize_nvfp4(x: torch.Tensor, per_tensor_scale: torch.Tensor, epsilon: float, pad_16x: bool,
                       hi_first: bool) -> tuple[torch.Tensor, torch.Tensor]:
    return _impl("quantize_nvfp4", {"x": x, "per_tensor_scale": per_tensor_scale, "epsilon": epsilon,
                                    "pad_16x": pad_16x, "hi_first": hi_first})


@_op_quantize_nvfp4.register_fake
def _(x, per_tensor_scale, epsilon, pad_16x, hi_first):
    rows, cols = x.shape
    if pad_16x:
        rows, cols = roundup(rows, 16), roundup(cols, 16)
    return (x.new_empty((rows, cols // 2), dtype=torch.uint8),
            x.new_empty((roundup(rows, 128), roundup(cols // 16, 4)), dtype=torch.float8_e4m3fn))


@torch.library.custom_op("comfy_kitchen::dequantize_nvfp4", mutates_args=())
def _op_dequantize_nvfp4(qx: torch.Tensor, per_tensor_scale: torch.Tensor, block_scales: torch.Tensor,
                         output_dtype_code: int, hi_first: bool) -> torch.Tensor:
    return _impl("dequantize_nvfp4", {"qx": qx, "per_tensor_scale": per_tensor_scale, "block_scales": block_scales,
                                      "output_type": DTYPE_CODE_TO_DTYPE[output_dtype_code], "hi_first": hi_first})


@_op_dequantize_nvfp4.register_fake
def _(qx, per_tensor_scale, block_scales, output_dtype_code, hi_first):
    rows, packed = qx.shape
    return qx.new_empty((rows, packed * 2), dtype=DTYPE_CODE_TO_DTYPE[output_dtype_code])


@torch.library.custom_op("comfy_kitchen::scaled_mm_nvfp4", mutates_args=())
def _op_scaled_mm_nvfp4(a: torch.Tensor, b: torch.Tensor, tensor_scale_a: torch.Tensor, tensor_scale_b: torch.Tensor,
                        block_scale_a: torch.Tensor, block_scale_b: torch.Tensor, bias: torch.Tensor | None,
                        output_dtype_code: int, alpha: torch.Tensor | None) -> torch.Tensor:
    return _impl("scaled_mm_nvfp4", {
        "a": a, "b": b, "tensor_scale_a": tensor_scale_a, "tensor_scale_b": tensor_scale_b,
        "block_scale_a": block_scale_a, "block_scale_b": block_scale_b, "bias": bias,
        "out_dtype": DTYPE_CODE_TO_DTYPE[output_dtype_code], "alpha": alpha})


@_op_scaled_mm_nvfp4.register_fake
def _(a, b, tensor_scale_a, tensor_scale_b, block_scale_a, block_scale_b, bias, output_dtype_code, alpha):
    return a.new_empty((a.shape[0], b.shape[0]), dtype=DTYPE_CODE_TO_DTYPE[output_dtype_code])


@torch.library.custom_op("comfy_kitchen::quantize_mxfp8", mutates_args=())
def _op_quantize_mxfp8(x: torch.Tensor, pad_32x: bool) -> tuple[torch.Tensor, torch.Tensor]:
    return _impl("quantize_mxfp8", {"x": x, "pad_32x": pad_32x})


@_op_quantize_mxfp8.register_fake
def _(x, pad_32x):
    rows, cols = x.shape
    if pad_32x:
        rows, cols = roundup(rows, 32), roundup(cols, 32)
    return (x.new_empty((rows, cols), dtype=torch.float8_e4m3fn),
            x.new_empty((roundup(rows, 128), roundup(cols // 32, 4)), dtype=torch.float8_e8m0fnu))


@torch.library.custom_op("comfy_kitchen::dequantize_mxfp8", mutates_args=())
def _op_dequantize_mxfp8(qx: torch.Tensor, block_scales: torch.Tensor, output_dtype_code: int) -> torch.Tensor:
    return _impl("dequantize_mxfp8", {"qx": qx, "block_scales": block_scales,
                                      "output_type": DTYPE_CODE_TO_DTYPE[output_dtype_code]})


@_op_dequantize_mxfp8.register_fake
def _(qx, block_scales, output_dtype_code):
    return torch.empty_like(qx, dtype=DTYPE_CODE_TO_DTYPE[output_dtype_code])


@torch.library.custom_op("comfy_kitchen::scaled_mm_mxfp8", mutates_args=())
def _op_scaled_mm_mxfp8(a: torch.Tensor, b: torch.Tensor, block_scale_a: torch.Tensor, block_scale_b: torch.Tensor,
                        bias: torch.Tensor | None, output_dtype_code: int) -> torch.Tensor:
    return _impl("scaled_mm_mxfp8", {"a": a, "b": b, "block_scale_a": block_scale_a, "block_scale_b": block_scale_b,
                                     "bias": bias, "out_dtype": DTYPE_CODE_TO_DTYPE[output_dtype_code]})


@_op_scaled_mm_mxfp8.register_fake
def _(a, b, block_scale_a, block_scale_b, bias, output_dtype_code):
    return a.new_empty((a.shape[0], b.shape[0]), dtype=DTYPE_CODE_TO_DTYPE[output_dtype_code])


if _registrations is not None and hasattr(_op_quantize_nvfp4, "_backend_fns") and hasattr(_op_quantize_nvfp4, "_disabled_kernel"):
    for _op in (_op_quantize_nvfp4, _op_dequantize_nvfp4, _op_scaled_mm_nvfp4, _op_quantize_mxfp8, _op_dequantize_mxfp8,
                _op_scaled_mm_mxfp8):
        _remember(_op)
