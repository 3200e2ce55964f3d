"""LM head fused with the cross-entropy loss.

The reference materialises fp32 logits ``[tokens, vocab]`` and runs max, exp,
sum, log, gather, mean as separate ops (implementation/nnfunctions.py:56-64,
layers.py:415-417).  Here the head GEMM writes bf16 logits, one kernel (rows up
to 32768 entries read once and written once) turns them into the loss and, in
place, into ``dlogits``, and two more GEMMs consume those: ``dh = dlogits W``
and ``dW += dlogitsᵀ h``.

Where the factor that the caller will back-propagate into the loss is known
(``grad_scale``; the pipeline step passes ``1 / microbatches``) and the weight
has a ``main_grad`` buffer, all of it happens in the forward pass, a chunk of
tokens at a time: no full logits tensor exists, and what is kept for the
backward pass is ``dh`` ``[tokens, d_model]``.  The backward pass multiplies
``dh`` by ``dloss / grad_scale``, which is one when the caller keeps its word
(in place, unless the graph is retained for another pass); the weight gradient
has already been accumulated with ``grad_scale``, once whatever follows.

Where it is not known, the forward pass keeps ``d(mean loss)/dlogits`` of as many
tokens as ``KEEP_BYTES`` hold, and the backward pass is two products over them
whose epilogues multiply by ``dloss``; the logits of the chunks beyond are
rebuilt.  Where no backward pass can follow, only the loss is formed, chunk by
chunk.  The value returned is the mean over tokens, like the reference.
"""
from __future__ import annotations

import torch

from . import backward_follows, cpp_nodes, functional as Fn, native, use_native

CHUNK_TOKENS = 4096
# Keeping logits saves one of four products and a pass over them for each token kept (6001 tokens, width 2048, 32000
# entries: 3307 us rebuilt, 2054 kept).  1 GiB is what a planned stage sets aside for the head's transients
# (parallel.memory: two logits tensors of a microbatch) at 8192 tokens of 32000 entries.
KEEP_BYTES = 1 << 30


def _chunks(first: int, total: int, size: int):
    for lo in range(first, total, size):
        yield lo, min(total, lo + size)


def _kept_tokens(tokens: int, vocab: int) -> int:
    """How many of ``tokens`` rows of bf16 logits ``KEEP_BYTES`` hold: all, or as many whole chunks as fit."""
    fit = KEEP_BYTES // (2 * vocab)
    return tokens if tokens <= fit else fit // CHUNK_TOKENS * CHUNK_TOKENS


class _LMHeadCE(torch.autograd.Function):
    @staticmethod
    def forward(ctx, hidden, weight, targets, grad_scale, wants_grad):
        h2d = hidden.reshape(-1, hidden.shape[-1])
        flat_targets = targets.reshape(-1).contiguous()
        tokens = h2d.shape[0]
        main_grad = getattr(weight, "main_grad", None)
        eager = wants_grad and grad_scale is not None and main_grad is not None and ctx.needs_input_grad[0]
        loss = torch.zeros((), dtype=torch.float64, device=hidden.device)
        ctx.weight, ctx.shape, ctx.eager, ctx.grad_scale = weight, hidden.shape, eager, grad_scale
        ctx.kept = _kept_tokens(tokens, weight.shape[0]) if wants_grad and not eager else 0
        kept = None
        if ctx.kept:
            kept = native.gemm_nt(h2d[:ctx.kept], weight)
            native.cross_entropy_scaled_(kept, flat_targets[:ctx.kept], loss, 1.0 / tokens, 1.0 / tokens)
        dh = torch.empty_like(h2d) if eager else None
        for lo, hi in _chunks(ctx.kept, tokens, CHUNK_TOKENS):
            logits = native.gemm_nt(h2d[lo:hi], weight)
            native.cross_entropy_scaled_(logits, flat_targets[lo:hi], loss, 1.0 / tokens,
                                         (grad_scale if eager else 1.0) / tokens)
            if eager:
                native.gemm_nn(logits, weight, out=dh[lo:hi])
                native.gemm_tn(logits, h2d[lo:hi], out=main_grad, accumulate=True)
        if eager:
            ctx.save_for_backward(dh)
        else:
            ctx.save_for_backward(h2d, flat_targets, kept)
        return loss.float()

    @staticmethod
    def backward(ctx, dloss):
        weight = ctx.weight
        if ctx.eager:
            (dh,) = ctx.saved_tensors
            if torch._C._autograd._get_current_graph_task_keep_graph():
                dh = dh.clone()          # a later backward pass through this graph scales what the forward pass left
            native.scale_(dh, dloss / ctx.grad_scale)
            return dh.view(ctx.shape), None, None, None, None
        h2d, flat_targets, kept = ctx.saved_tensors
        tokens = h2d.shape[0]
        scale = dloss.to(device=h2d.device, dtype=torch.float32)
        main_grad = getattr(weight, "main_grad", None)
        wants_dw = main_grad is not None or ctx.needs_input_grad[1]
        whole = 0 < tokens == ctx.kept
        dh = torch.empty_like(h2d) if ctx.needs_input_grad[0] else None
        dw = main_grad
        if wants_dw and main_grad is None and not whole:
            dw = torch.zeros(weight.shape, dtype=torch.float32, device=weight.device)
        if ctx.kept:
            if dh is not None:
                native.gemm_nn(kept, weight, out=dh[:ctx.kept], alpha=scale)
            if wants_dw and dw is None:
                dw = native.gemm_tn(kept, h2d, out_dtype=weight.dtype, alpha=scale)
            elif wants_dw:
                native.gemm_tn(kept, h2d[:ctx.kept], out=dw, accumulate=True, alpha=scale)
        scratch = torch.zeros((), dtype=torch.float32, device=h2d.device)
        for lo, hi in _chunks(ctx.kept, tokens, CHUNK_TOKENS):
            logits = native.gemm_nt(h2d[lo:hi], weight)
            native.cross_entropy_scaled_(logits, flat_targets[lo:hi], scratch, 1.0 / tokens, 1.0 / tokens)
            native.scale_(logits, dloss)
            if dh is not None:
                native.gemm_nn(logits, weight, out=dh[lo:hi])
            if wants_dw:
                native.gemm_tn(logits, h2d[lo:hi], out=dw, accumulate=True)
        return (None if dh is None else dh.view(ctx.shape), None if main_grad is not None or dw is None
                else dw.to(weight.dtype), None, None, None)


def lm_head_cross_entropy(hidden: torch.Tensor, weight: torch.Tensor, targets: torch.Tensor,
                          grad_scale: float | None = None) -> torch.Tensor:
    """Mean next-token loss of ``hidden @ weightᵀ`` against ``targets``.  ``grad_scale``: the factor the caller will
    back-propagate into the returned loss, when it is known in advance (see the module text)."""
    from .dense import linear
    if use_native(hidden, "lmhead_ce"):
        grad = getattr(weight, "main_grad", None)
        if grad is not None and grad_scale is not None:
            nodes = cpp_nodes(hidden, weight, targets, grad)
            loss = nodes.head(hidden, weight, targets, grad, grad_scale, CHUNK_TOKENS, native.status_word(hidden.device)) \
                if nodes else None
            if loss is not None:
                return loss
        return _LMHeadCE.apply(hidden, weight, targets, grad_scale, backward_follows(hidden, weight))
    logits = linear(hidden, weight)
    return Fn.cross_entropy(logits.reshape(-1, logits.shape[-1]), targets.reshape(-1))
