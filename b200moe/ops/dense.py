"""Linear, embedding and RMSNorm ops with explicit backward passes.

Weight gradients follow the "main grad" convention: when the weight tensor
carries a ``main_grad`` attribute (an fp32 buffer owned by the FSDP wrapper)
the backward pass accumulates ``dW`` straight into it from the GEMM epilogue
and returns no gradient to autograd.  Otherwise the gradient is returned and
autograd accumulates it in ``.grad``.

Replaces the reference's ``einsum`` linear (implementation/layers.py:55-69),
``weight[x, :]`` embedding (layers.py:72-82) and fp32 RMSNorm (layers.py:84-97).
"""
from __future__ import annotations

import torch

from . import backward_follows, cpp_nodes, functional as Fn, native, use_native


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, rope=None):
        """``rope``: optional ``(cos, sin, rope_cols, seq)``: the rotary embedding is applied to the leading
        ``rope_cols`` output columns in the GEMM epilogue.  The backward pass then expects the gradient of the
        UNROTATED output (the attention backward kernels deliver exactly that)."""
        ctx.weight = weight
        ctx.save_for_backward(x)
        x2d = x.reshape(-1, x.shape[-1])
        # a weight whose peer rows have not arrived yet carries the call that gathers them and multiplies in one
        # kernel (set by the FSDP wrapper after an optimizer step, consumed by the first use)
        gather = getattr(weight, "pending_gather", None)
        if gather is not None:
            weight.pending_gather = None
            y = gather(x2d if x2d.is_contiguous() else x2d.contiguous())
            if rope is not None:
                cos, sin, cols, seq = rope
                native.rope_inplace(y, 0, y.shape[0], seq, cols // 128, 128, y.shape[1], cos, sin, 1.0)
        elif rope is not None:
            cos, sin, cols, seq = rope
            y = native.gemm_nt_rope(x2d, weight, cos, sin, cols, seq)
        elif use_native(x, "gemm"):
            y = native.gemm_nt(x2d, weight)
        else:
            w = weight if weight.dtype == x.dtype else weight.to(x.dtype)
            y = x2d @ w.t()
        return y if x.dim() == 2 else y.view(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        (x,) = ctx.saved_tensors
        weight = ctx.weight
        x2d = x.reshape(-1, x.shape[-1])
        dy2d = dy.reshape(-1, dy.shape[-1])
        if not dy2d.is_contiguous():
            dy2d = dy2d.contiguous()
        on_gpu = use_native(x, "gemm")
        dx = None
        if ctx.needs_input_grad[0]:
            if on_gpu:
                dx = native.gemm_nn(dy2d, weight)
            else:
                w = weight if weight.dtype == dy2d.dtype else weight.to(dy2d.dtype)
                dx = dy2d @ w
            dx = dx.view_as(x)
        dw = None
        main_grad = getattr(weight, "main_grad", None)
        if main_grad is not None:
            if on_gpu:
                native.gemm_tn(dy2d, x2d, out=main_grad, accumulate=True)
            else:
                main_grad.addmm_(dy2d.t().to(main_grad.dtype), x2d.to(main_grad.dtype))
        elif ctx.needs_input_grad[1]:
            if on_gpu:
                dw = native.gemm_tn(dy2d, x2d, out_dtype=weight.dtype)
            else:
                dw = (dy2d.t() @ x2d).to(weight.dtype)
        return dx, dw, None


def linear(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``y = x @ weightᵀ`` with ``weight`` of shape ``[d_out, d_in]``; no bias."""
    return _Linear.apply(x, weight)


def linear_rope(x: torch.Tensor, weight: torch.Tensor, cos, sin, rope_cols: int, seq: int) -> torch.Tensor:
    """GPU only: ``x @ weightᵀ`` (``x [tokens, d_in]``, tokens laid out as sequences of ``seq``) with the rotary
    embedding (heads of 128 columns, adjacent pairs) applied to output columns ``[0, rope_cols)`` inside the GEMM.
    Its backward pass takes the gradient with respect to the unrotated product."""
    return _Linear.apply(x, weight, (cos[:seq].contiguous(), sin[:seq].contiguous(), rope_cols, seq))


class _SwiGLUFFN(torch.autograd.Function):
    """``(silu(x W1ᵀ) · (x W3ᵀ)) W2ᵀ``: gate/up product with the SwiGLU in its epilogue and the down projection;
    backward: ``dh`` product with the SwiGLU backward in its epilogue, ``dx`` over the concatenated reduction, three
    weight gradients."""

    @staticmethod
    def forward(ctx, x, w1, w3, w2, keep):
        x2d = x.reshape(-1, x.shape[-1])
        h, gate, up = native.gemm_swiglu(x2d, w1.unsqueeze(0), w3.unsqueeze(0), save_gate_up=keep)
        y = native.gemm_nt(h, w2)
        ctx.weights = (w1, w3, w2)
        if keep:
            ctx.save_for_backward(x, gate, up)
        return y.view(*x.shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, gate, up = ctx.saved_tensors
        w1, w3, w2 = ctx.weights
        x2d, ffn = x.reshape(-1, x.shape[-1]), w1.shape[0]
        dy2d = dy.reshape(-1, dy.shape[-1]).contiguous()
        dgu, h = native.gemm_nn_swiglu_bwd(dy2d, w2, gate, up)
        dx = native.gemm_nn(dgu, w1, w2=w3).view_as(x) if ctx.needs_input_grad[0] else None
        grads = [None, None, None]
        accumulators = [getattr(w, "main_grad", None) for w in ctx.weights]
        first = 0
        if accumulators[0] is accumulators[1] is None and all(ctx.needs_input_grad[1:3]):
            grads[0], grads[1] = torch.empty_like(w1), torch.empty_like(w3)
            native.gemm_tn_two(dgu, x2d, grads[0], grads[1], False)      # both weights read x: one launch
            first = 2
        products = ((dgu[:, :ffn], x2d), (dgu[:, ffn:], x2d), (dy2d, h))
        for i in range(first, 3):
            left, right = products[i]
            if accumulators[i] is not None:
                native.gemm_tn(left, right, out=accumulators[i], accumulate=True)
            elif ctx.needs_input_grad[i + 1]:
                grads[i] = native.gemm_tn(left, right, out_dtype=ctx.weights[i].dtype)
        return dx, *grads, None


def swiglu_ffn(x, w1, w3, w2):
    """The dense SwiGLU layer on the fused kernels, or ``None`` where its three products have to run one by one: CPU,
    other types, a weight that is still to be gathered, layouts and widths that the fused epilogues do not tile (they
    take 128 gate columns beside 128 up columns, and reduce in steps of 64).  4096 x 4096 -> 14336, forward and
    backward: 3.5 ms instead of 5.2, of which 1.6 were elementwise passes over the hidden layer."""
    weights = (w1, w3, w2)
    if not (use_native(x, "gemm") and use_native(x, "swiglu") and x.dtype == torch.bfloat16 and x.numel() > 0
            and x.data_ptr() % 16 == 0 and x.is_contiguous() and all(
                w.dtype == torch.bfloat16 and w.dim() == 2 and w.is_contiguous() and w.data_ptr() % 16 == 0
                and w.device == x.device and getattr(w, "pending_gather", None) is None for w in weights)):
        return None
    ffn, dim = w1.shape
    if w3.shape != w1.shape or w2.shape != (dim, ffn) or ffn % 128 or dim % 64 or x.shape[-1] != dim:
        return None
    return _SwiGLUFFN.apply(x, *weights, backward_follows(x, *weights))


class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, table):
        ctx.table = table
        ctx.save_for_backward(ids)
        if use_native(table, "embedding"):
            return native.embedding_fwd(ids, table)
        return table[ids]

    @staticmethod
    def backward(ctx, dy):
        (ids,) = ctx.saved_tensors
        table = ctx.table
        flat_ids = ids.reshape(-1)
        dy2d = dy.reshape(-1, dy.shape[-1])
        main_grad = getattr(table, "main_grad", None)
        if main_grad is not None:
            if use_native(dy, "embedding"):
                native.embedding_bwd(flat_ids, dy2d, main_grad)
            else:
                main_grad.index_add_(0, flat_ids, dy2d.to(main_grad.dtype))
            return None, None
        grad = torch.zeros_like(table, dtype=torch.float32)
        grad.index_add_(0, flat_ids, dy2d.float())
        return None, grad.to(table.dtype)


def embedding(ids: torch.Tensor, table: torch.Tensor) -> torch.Tensor:
    """Row gather ``table[ids]``; the backward pass scatter-adds in fp32."""
    grad = getattr(table, "main_grad", None)
    if grad is not None and use_native(table, "embedding"):
        nodes = cpp_nodes(ids, table, grad)
        out = nodes.embedding(ids, table, grad) if nodes else None
        if out is not None:
            return out
    return _Embedding.apply(ids, table)


class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, eps):
        y, rstd = native.rmsnorm_fwd(x, weight, eps)
        ctx.save_for_backward(x, weight, rstd)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, rstd = ctx.saved_tensors
        dx, dw = native.rmsnorm_bwd(dy.contiguous(), x, weight, rstd)
        return dx, dw.to(weight.dtype), None


def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-5) -> torch.Tensor:
    """``x · rsqrt(mean(x²) + eps) · weight`` evaluated in fp32, cast back."""
    if use_native(x, "rmsnorm"):
        nodes = cpp_nodes(x, weight)
        out = nodes.rmsnorm(x, weight, eps, native.status_word(x.device)) if nodes else None
        return _RMSNorm.apply(x, weight, eps) if out is None else out
    return Fn.rmsnorm_ref(x, weight, eps)


class _AddRMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, weight, eps):
        summed, y, rstd = native.add_rmsnorm_fwd(x, delta, weight, eps)
        ctx.save_for_backward(summed, weight, rstd)
        return summed, y

    @staticmethod
    def backward(ctx, dsum, dy):
        summed, weight, rstd = ctx.saved_tensors
        dx, dw = native.rmsnorm_bwd(dy.contiguous(), summed, weight, rstd, residual_grad=dsum)
        return dx, dx, dw.to(weight.dtype), None


def add_rmsnorm(x: torch.Tensor, delta: torch.Tensor, weight: torch.Tensor, eps: float = 1e-5):
    """Residual add fused with the following norm: returns ``(x + delta,
    rmsnorm(x + delta))``."""
    if use_native(x, "rmsnorm"):
        return _AddRMSNorm.apply(x, delta, weight, eps)
    summed = x + delta
    return summed, Fn.rmsnorm_ref(summed, weight, eps)
