"""Operator seams of the model.

Every hot op of the training step is a function here.  On a CUDA tensor the
function launches the hand-written sm_100a kernel from the in-tree extension
(``b200moe/ops/native.py`` loads it and raises if it is missing on a GPU box);
on a CPU tensor it evaluates the plain PyTorch statement from
``b200moe.ops.functional``, which is the oracle the kernels are tested against
and the compute path of the CPU/gloo plumbing tier.

``set_native(False)`` forces the PyTorch statements on CUDA tensors too; it is an
A/B switch for tests and for the library-kernel baseline measurement, not a
product path.
"""
from __future__ import annotations

import os

import torch

from . import functional as Fn

_FORCE_TORCH = os.environ.get("B200MOE_NATIVE", "1") == "0"
_DISABLED: set[str] = set(filter(None, os.environ.get("B200MOE_DISABLE", "").split(",")))


def set_native(enabled: bool) -> None:
    global _FORCE_TORCH
    _FORCE_TORCH = not enabled


def native_enabled() -> bool:
    return not _FORCE_TORCH


def use_native(t: torch.Tensor, op: str = "") -> bool:
    """True when ``t`` lives on a GPU and native kernels are switched on."""
    if not t.is_cuda or _FORCE_TORCH or op in _DISABLED:
        return False
    from . import native
    return native.has(op)


def cpp_nodes(*tensors):
    """The C++ autograd nodes for these operands, or ``None``: they take plain tensors outside of every transformation that
    looks through Python nodes (function transforms, forward-mode differentiation, tracing)."""
    from torch.autograd import forward_ad
    from . import native
    if (any(type(t) is not torch.Tensor and type(t) is not torch.nn.Parameter for t in tensors)
            or torch._C._are_functorch_transforms_active() or forward_ad._current_level >= 0
            or torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.overrides._get_current_function_mode_stack()
            or torch.utils._python_dispatch._get_current_dispatch_mode() is not None):
        return None
    return native.nodes()


def backward_follows(*tensors) -> bool:
    """Whether a call on ``tensors`` (``None`` among them) can be differentiated.  Asked by the callers of autograd
    functions: inside ``forward`` grad mode is off, and ``ctx.needs_input_grad`` repeats the inputs' ``requires_grad``
    even under ``no_grad``."""
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


from .dense import linear, linear_rope, swiglu_ffn, embedding, rmsnorm, add_rmsnorm  # noqa: E402
from .attention import rope_attention  # noqa: E402
from .loss import lm_head_cross_entropy  # noqa: E402
from .moe import router_top2, moe_ffn, DispatchPlan  # noqa: E402

__all__ = [
    "Fn", "set_native", "native_enabled", "use_native", "backward_follows", "linear", "linear_rope", "swiglu_ffn",
    "embedding", "rmsnorm", "add_rmsnorm",
    "rope_attention", "lm_head_cross_entropy", "router_top2", "moe_ffn", "DispatchPlan",
]
