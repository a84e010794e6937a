"""Declarative argument constraints checked before a backend is chosen.

Public names and semantics follow the reference's comfy_kitchen/constraints.py:30-250
(shape rules, per-parameter dtype/device/shape constraints, per-function device set
and minimum compute capability, first-failure validation result).
"""
from __future__ import annotations

from collections.abc import Mapping
from dataclasses import dataclass, field

import torch

__all__ = [
    "DivisibleBy",
    "ExactDims",
    "FunctionConstraints",
    "MinDims",
    "ParamConstraint",
    "ShapeRule",
    "ValidationResult",
    "validate_function_call",
    "validate_param",
]


class ShapeRule:
    """A predicate over a tensor's shape with a printable description."""

    def check(self, tensor: torch.Tensor) -> bool:  # pragma: no cover - interface
        raise NotImplementedError

    def describe(self) -> str:  # pragma: no cover - interface
        raise NotImplementedError


@dataclass(frozen=True)
class DivisibleBy(ShapeRule):
    dim: int
    factor: int

    def check(self, tensor: torch.Tensor) -> bool:
        return tensor.dim() > self.dim and tensor.shape[self.dim] % self.factor == 0

    def describe(self) -> str:
        return f"dim[{self.dim}] divisible by {self.factor}"


@dataclass(frozen=True)
class MinDims(ShapeRule):
    ndim: int

    def check(self, tensor: torch.Tensor) -> bool:
        return tensor.dim() >= self.ndim

    def describe(self) -> str:
        return f"at least {self.ndim}D"


@dataclass(frozen=True)
class ExactDims(ShapeRule):
    ndim: int

    def check(self, tensor: torch.Tensor) -> bool:
        return tensor.dim() == self.ndim

    def describe(self) -> str:
        return f"exactly {self.ndim}D"


@dataclass(frozen=True)
class ParamConstraint:
    """Allowed dtypes / device types / shapes of one keyword argument (None = any)."""

    dtypes: frozenset[torch.dtype] | None = None
    devices: frozenset[str] | None = None
    shape_rules: tuple[ShapeRule, ...] = ()

    def check_dtype(self, value) -> bool:
        if self.dtypes is None:
            return True
        dt = value.dtype if isinstance(value, torch.Tensor) else value
        return dt in self.dtypes

    def check_device(self, tensor: torch.Tensor, default_devices: frozenset[str]) -> bool:
        allowed = default_devices if self.devices is None else self.devices
        return "*" in allowed or tensor.device.type in allowed

    def check_shape(self, tensor: torch.Tensor) -> bool:
        return all(r.check(tensor) for r in self.shape_rules)

    def accepts(self, value, default_devices: frozenset[str]) -> bool:
        """All three checks (of a value that is not a tensor: its dtype alone)."""
        if not isinstance(value, torch.Tensor):
            return self.dtypes is None or value in self.dtypes
        if self.dtypes is not None and value.dtype not in self.dtypes:
            return False
        allowed = default_devices if self.devices is None else self.devices
        if not (value.is_cuda and "cuda" in allowed) and "*" not in allowed and value.device.type not in allowed:
            return False
        for rule in self.shape_rules:
            if not rule.check(value):
                return False
        return True


@dataclass(frozen=True)
class FunctionConstraints:
    params: dict[str, ParamConstraint] = field(default_factory=dict)
    default_devices: frozenset[str] = field(default_factory=lambda: frozenset({"cuda", "cpu"}))
    min_compute_capability: tuple[int, int] | None = None

    def __hash__(self) -> int:
        return hash((tuple(sorted(self.params.items(), key=lambda kv: kv[0])), self.default_devices,
                     self.min_compute_capability))


@dataclass
class ValidationResult:
    success: bool
    failed_param: str | None = None
    failure_reason: str | None = None

    @staticmethod
    def ok() -> "ValidationResult":
        return ValidationResult(True)

    @staticmethod
    def fail(param: str, reason: str) -> "ValidationResult":
        return ValidationResult(False, param, reason)


def validate_param(name, value, constraint: ParamConstraint, default_devices: frozenset[str]) -> ValidationResult:
    """Check one argument; ``None`` always passes, a bare dtype is checked against ``dtypes`` only."""
    if value is None:
        return ValidationResult.ok()
    if not constraint.check_dtype(value):
        dt = value.dtype if isinstance(value, torch.Tensor) else value
        return ValidationResult.fail(name, f"dtype {dt} not in {set(constraint.dtypes)}")
    if not isinstance(value, torch.Tensor):
        return ValidationResult.ok()
    if not constraint.check_device(value, default_devices):
        allowed = default_devices if constraint.devices is None else constraint.devices
        return ValidationResult.fail(name, f"device {value.device.type} not in {set(allowed)}")
    for rule in constraint.shape_rules:
        if not rule.check(value):
            return ValidationResult.fail(name, f"shape {list(value.shape)} fails: {rule.describe()}")
    return ValidationResult.ok()


def validate_function_call(constraints: FunctionConstraints, kwargs: Mapping, compute_capability=None) -> ValidationResult:
    """Hardware gate first, then every constrained argument in declaration order."""
    need = constraints.min_compute_capability
    if need is not None:
        if compute_capability is None:
            return ValidationResult.fail("__hardware__", "CUDA compute capability required but not available")
        if compute_capability != need and tuple(compute_capability) < tuple(need):
            return ValidationResult.fail(
                "__hardware__",
                f"compute capability {compute_capability[0]}.{compute_capability[1]} < required {need[0]}.{need[1]}")
    for pname, pc in constraints.params.items():
        value = kwargs.get(pname)
        if value is None or pc.accepts(value, constraints.default_devices):
            continue
        return validate_param(pname, value, pc, constraints.default_devices)  # says what failed
    return ValidationResult.ok()
