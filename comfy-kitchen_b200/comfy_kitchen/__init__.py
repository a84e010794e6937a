"""comfy_kitchen operator API backed by a single sm_100a (B200) C-ABI library.

Function names, signatures, defaults and return shapes/dtypes follow the reference's
comfy_kitchen/__init__.py:118-272 and :311-366 for the quantized-linear path:
``quantize_nvfp4``, ``scaled_mm_nvfp4``, ``quantize_mxfp8``, ``scaled_mm_mxfp8`` and the
backend-configuration calls.  Every operator goes through its
``torch.ops.comfy_kitchen.*`` custom op (eager calls on plain CUDA tensors, to which that layer
adds nothing while nobody has registered a kernel of their own, straight) to the one registered backend;
there is no CPU implementation behind these calls.
"""
from __future__ import annotations

import torch

from . import ops as _ops  # noqa: F401  (defines torch.ops.comfy_kitchen.*)
from .backends import cuda as _cuda_backend  # noqa: F401
from .backends import eager as _eager_backend  # noqa: F401
from .backends import triton as _triton_backend  # noqa: F401
from .exceptions import BackendError, BackendNotFoundError, BackendNotImplementedError, NoCapableBackendError
from .float_utils import from_blocked, swap_nibbles, to_blocked
from .ops import DTYPE_TO_CODE, _impl, dispatcher_adds_nothing, host_operator, replaced
from .registry import registry

__version__ = "0.1.0"

__all__ = [
    "quantize_nvfp4",
    "dequantize_nvfp4",
    "quantize_mxfp8",
    "dequantize_mxfp8",
    "scaled_mm_nvfp4",
    "scaled_mm_mxfp8",
    "swap_nibbles",
    "to_blocked",
    "from_blocked",
    "list_backends",
    "set_backend_priority",
    "enable_backend",
    "disable_backend",
    "use_backend",
    "BackendError",
    "BackendNotFoundError",
    "BackendNotImplementedError",
    "NoCapableBackendError",
]


def quantize_nvfp4(x: torch.Tensor, per_tensor_scale: torch.Tensor, epsilon: float = 0.0, pad_16x: bool = False,
                   hi_first: bool = True) -> tuple[torch.Tensor, torch.Tensor]:
    """Quantize a 2-D tensor to NVFP4.

    Returns ``(codes, block_scales)``: packed E2M1 codes ``uint8 [M', K'/2]`` and E4M3
    scales of 16-element blocks ``float8_e4m3fn [roundup(M',128), roundup(K'/16,4)]`` in
    the swizzled tensor-core layout.  With ``pad_16x`` both dimensions are zero-padded
    to multiples of 16.  ``hi_first`` puts the even-indexed element of each pair in the
    high nibble.  ``epsilon`` is unused (kept for signature compatibility).
    """
    host = host_operator("quantize_nvfp4")
    if host is not None and type(epsilon) is float:
        out = host(x, per_tensor_scale, pad_16x, hi_first)
        if out is not None:
            return out
    if not replaced("quantize_nvfp4") and dispatcher_adds_nothing((x, per_tensor_scale)) and type(epsilon) is float and \
            type(pad_16x) is bool and type(hi_first) is bool:
        return _impl("quantize_nvfp4", {"x": x, "per_tensor_scale": per_tensor_scale, "epsilon": epsilon, "pad_16x": pad_16x,
                                        "hi_first": hi_first})
    return torch.ops.comfy_kitchen.quantize_nvfp4(x, per_tensor_scale, epsilon, pad_16x, hi_first)


def dequantize_nvfp4(qx: torch.Tensor, per_tensor_scale: torch.Tensor, block_scales: torch.Tensor,
                     output_type: torch.dtype = torch.bfloat16, hi_first: bool = True) -> torch.Tensor:
    """Inverse of :func:`quantize_nvfp4` into ``output_type`` (float32, float16 or bfloat16)."""
    code = DTYPE_TO_CODE[output_type]
    host = host_operator("dequantize_nvfp4")
    if host is not None:
        out = host(qx, per_tensor_scale, block_scales, output_type, hi_first)
        if out is not None:
            return out
    if not replaced("dequantize_nvfp4") and dispatcher_adds_nothing((qx, per_tensor_scale, block_scales)) and type(hi_first) is bool:
        return _impl("dequantize_nvfp4", {"qx": qx, "per_tensor_scale": per_tensor_scale, "block_scales": block_scales,
                                          "output_type": output_type, "hi_first": hi_first})
    return torch.ops.comfy_kitchen.dequantize_nvfp4(qx, per_tensor_scale, block_scales, code, hi_first)


def scaled_mm_nvfp4(a: torch.Tensor, b: torch.Tensor, tensor_scale_a: torch.Tensor, tensor_scale_b: torch.Tensor,
                    block_scale_a: torch.Tensor, block_scale_b: torch.Tensor, bias: torch.Tensor | None = None,
                    out_dtype: torch.dtype | None = None, alpha: torch.Tensor | None = None) -> torch.Tensor:
    """``(a @ b.T) * (tensor_scale_a * tensor_scale_b) + bias`` on NVFP4 operands; ``[M, N]`` in ``out_dtype`` (bf16 by default)."""
    if out_dtype is None:
        out_dtype = torch.bfloat16
    code = DTYPE_TO_CODE[out_dtype]
    host = host_operator("scaled_mm_nvfp4")
    if host is not None:
        out = host(a, b, tensor_scale_a, tensor_scale_b, block_scale_a, block_scale_b, bias, out_dtype, alpha)
        if out is not None:
            return out
    if not replaced("scaled_mm_nvfp4") and \
            dispatcher_adds_nothing((a, b, tensor_scale_a, tensor_scale_b, block_scale_a, block_scale_b), (bias, alpha)):
        return _impl("scaled_mm_nvfp4", {
            "a": a, "b": b, "tensor_scale_a": tensor_scale_a, "tensor_scale_b": tensor_scale_b, "block_scale_a": block_scale_a,
            "block_scale_b": block_scale_b, "bias": bias, "out_dtype": out_dtype, "alpha": alpha})
    return torch.ops.comfy_kitchen.scaled_mm_nvfp4(a, b, tensor_scale_a, tensor_scale_b, block_scale_a, block_scale_b,
                                                   bias, code, alpha)


def quantize_mxfp8(x: torch.Tensor, pad_32x: bool = False) -> tuple[torch.Tensor, torch.Tensor]:
    """Quantize a 2-D tensor to MXFP8: ``(float8_e4m3fn [M', K'], float8_e8m0fnu swizzled scales of 32-element blocks)``."""
    host = host_operator("quantize_mxfp8")
    if host is not None:
        out = host(x, pad_32x)
        if out is not None:
            return out
    if not replaced("quantize_mxfp8") and dispatcher_adds_nothing((x,)) and type(pad_32x) is bool:
        return _impl("quantize_mxfp8", {"x": x, "pad_32x": pad_32x})
    return torch.ops.comfy_kitchen.quantize_mxfp8(x, pad_32x)


def dequantize_mxfp8(qx: torch.Tensor, block_scales: torch.Tensor,
                     output_type: torch.dtype = torch.bfloat16) -> torch.Tensor:
    """Inverse of :func:`quantize_mxfp8` into ``output_type``."""
    code = DTYPE_TO_CODE[output_type]
    host = host_operator("dequantize_mxfp8")
    if host is not None:
        out = host(qx, block_scales, output_type)
        if out is not None:
            return out
    if not replaced("dequantize_mxfp8") and dispatcher_adds_nothing((qx, block_scales)):
        return _impl("dequantize_mxfp8", {"qx": qx, "block_scales": block_scales, "output_type": output_type})
    return torch.ops.comfy_kitchen.dequantize_mxfp8(qx, block_scales, code)


def scaled_mm_mxfp8(a: torch.Tensor, b: torch.Tensor, block_scale_a: torch.Tensor, block_scale_b: torch.Tensor,
                    bias: torch.Tensor | None = None, out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """``a @ b.T + bias`` on MXFP8 operands; ``[M, N]`` in ``out_dtype`` (bf16 by default)."""
    if out_dtype is None:
        out_dtype = torch.bfloat16
    code = DTYPE_TO_CODE[out_dtype]
    host = host_operator("scaled_mm_mxfp8")
    if host is not None:
        out = host(a, b, block_scale_a, block_scale_b, bias, out_dtype)
        if out is not None:
            return out
    if not replaced("scaled_mm_mxfp8") and dispatcher_adds_nothing((a, b, block_scale_a, block_scale_b), (bias,)):
        return _impl("scaled_mm_mxfp8", {"a": a, "b": b, "block_scale_a": block_scale_a, "block_scale_b": block_scale_b,
                                         "bias": bias, "out_dtype": out_dtype})
    return torch.ops.comfy_kitchen.scaled_mm_mxfp8(a, b, block_scale_a, block_scale_b, bias, code)


# ---- backend configuration (comfy_kitchen/__init__.py:311-366 of the reference) ----------------
def set_backend_priority(priority: list[str]) -> None:
    registry.set_priority(priority)


def disable_backend(name: str) -> None:
    registry.disable(name)


def enable_backend(name: str) -> None:
    registry.enable(name)


def list_backends() -> dict:
    """``{name: {"available", "disabled", "unavailable_reason", "capabilities"}}`` for ``cuda``, ``eager`` and ``triton``."""
    return registry.list_backends()


def use_backend(name: str):
    """Context manager forcing one backend for the calling thread."""
    return registry.use_backend(name)
