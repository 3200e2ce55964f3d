"""The attention half of a block as one node: norm, fused projection with rotation, causal attention, output projection,
residual sum and the norm behind it (``AttnHalf`` in ``csrc/nodes.cpp``, the launches in ``csrc/layers.cu``), the kernels those of
the separate operations.  The two gradients of the block's input are summed by the norm's backward kernel instead of an
operation of their own.

Stands, for the operands and switches it takes, for the chain of ``ops.rmsnorm``, ``ops.linear_rope``,
``fused_qkv_attention``, ``ops.linear`` and ``ops.add_rmsnorm`` of ``TransformerLayer.forward``.
"""
from __future__ import annotations

from . import cpp_nodes, native, use_native
from .attention import attention_backend


def attn_half(x, ln1, wqkv, cos, sin, wo, ln2, heads, eps1, eps2):
    """``(x + attention(norm(x)), its norm)`` of ``x [B, S, D]``, or ``None`` where the operations have to run one by one: CPU,
    other types and layouts, sequences that are no multiple of 128, head sizes other than 128, weights that are still to be
    gathered or have no fp32 gradient buffer, kernels switched off, launches that are timed one by one."""
    gqkv, go = getattr(wqkv, "main_grad", None), getattr(wo, "main_grad", None)
    if (gqkv is None or go is None or getattr(wqkv, "pending_gather", None) is not None or getattr(wo, "pending_gather", None) is not None
            or not all(use_native(x, op) for op in ("rmsnorm", "gemm", "attention")) or attention_backend() != "native"):
        return None
    nodes = cpp_nodes(x, ln1, wqkv, gqkv, cos, sin, wo, go, ln2)
    return nodes.attn_half(x, ln1, wqkv, gqkv, cos, sin, wo, go, ln2, native.status_word(x.device), *heads, eps1, eps2) \
        if nodes else None
