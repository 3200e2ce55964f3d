"""The MoE block as native kernels with a hand-written backward pass.

One rank (``_MoEFused``): plan (device counting sort) → gather rows into the
padded expert-major buffer → grouped gate/up GEMM with the SwiGLU epilogue →
grouped down GEMM → weighted combine; backward: the duals in reverse, with the
three weight-gradient GEMMs accumulating into the experts' ``main_grad``
buffers.  An expert group of several ranks (``_MoEPull``): the row exchange is
part of the expert GEMMs (``b200moe.comm.ep``).  In both, no step involves the
host: tile counts, segment offsets and the tile→expert table stay on the device
and the persistent GEMMs read them there.

Replaces the reference's ``_dispatch_tokens`` / ``GroupedPositionWiseFFLayer`` /
``_combine_tokens`` (implementation/layers.py:139-246) including its per-expert
``nonzero`` loop and ``.cpu()`` split exchange.
"""
from __future__ import annotations

import torch

from . import backward_follows, cpp_nodes, native

ALIGN = 256       # expert segments are padded to 256 rows (whole 256x256 GEMM tiles)


def capacity_rows(slots: int, num_experts: int) -> int:
    """Worst-case rows of the padded expert-major buffer."""
    return (slots + num_experts * (ALIGN - 1) + ALIGN - 1) // ALIGN * ALIGN


def _wgrad(dy, x, param, offs, num_experts, counts=None):
    main = getattr(param, "main_grad", None)
    if main is not None:
        native.gemm_tn(dy, x, out=main, accumulate=True, expert_offsets=offs, num_experts=num_experts, counts=counts)
        return None
    return native.gemm_tn(dy, x, out_dtype=param.dtype, expert_offsets=offs, num_experts=num_experts, counts=counts)


def _wgrad_gate_up(dgu, x, w1, w3, offs, num_experts, counts):
    """Gradients of the gate and up weights, in one launch where their accumulators are alike."""
    ffn = w1.shape[1]
    one, two = getattr(w1, "main_grad", None), getattr(w3, "main_grad", None)
    if one is None and two is None and w1.dtype == w3.dtype == torch.bfloat16:
        grads = torch.empty(w1.shape, dtype=w1.dtype, device=dgu.device), torch.empty_like(w3, dtype=w3.dtype)
        native.gemm_tn_two(dgu, x, *grads, False, offs, num_experts, counts)
        return grads
    if (one is not None and two is not None and one.dtype == two.dtype and one.shape == two.shape
            and one.is_contiguous() and two.is_contiguous()):
        native.gemm_tn_two(dgu, x, one, two, True, offs, num_experts, counts)
        return None, None
    return (_wgrad(dgu[:, :ffn], x, w1, offs, num_experts, counts),
            _wgrad(dgu[:, ffn:], x, w3, offs, num_experts, counts))


def _experts_forward(x, weights, idx, w1, w2, w3, recompute, budget, wants_grad, residual=None):
    """Plan, gather, gate/up, down projection and combine.  Returns ``(out, recompute, ledger, saved)``; the last of
    ``saved`` are the experts' slot counts."""
    tokens, dim = x.shape
    experts = w1.shape[0]
    cap = capacity_rows(tokens * 2, experts)
    slot_row, row_slot, offs, tile_expert, meta, counts = native.moe_plan(idx, experts, cap)
    x_perm = native.moe_gather(x, row_slot, meta, cap)
    tiles = meta[0:1]
    # what this call keeps for its backward pass: the permuted input and the expert outputs always, the
    # gate/up pre-activations while the stage's activation budget has room for them
    ledger = None
    if budget is not None and wants_grad:
        ledger = (cap * dim * 4, cap * w1.shape[1] * 4)
        kept = budget.enter(*ledger)
        recompute = recompute or not kept
        ledger += (not recompute,)
    keep = wants_grad and not recompute
    h, gate, up = native.gemm_swiglu(x_perm, w1, w3, tile_expert, tiles, save_gate_up=keep, align256=True)
    y_perm = native.gemm_nt(h, w2, tile_expert=tile_expert, num_m_tiles=tiles, num_experts=experts, align256=True)
    out = native.moe_combine(y_perm, slot_row, weights, tokens, residual=residual)
    saved = [x_perm, y_perm, weights, offs, tile_expert, meta, slot_row, row_slot]
    if keep:
        saved += [gate, up]
    return out, recompute, ledger, saved + [counts]


def _experts_backward(dout, saved, counts, w1, w2, w3, recompute):
    """Returns ``(dx_perm, dweights, dw1, dw2, dw3)``."""
    x_perm, y_perm, weights, offs, tile_expert, meta, slot_row, row_slot = saved[:8]
    tokens, cap, experts = weights.shape[0], x_perm.shape[0], w1.shape[0]
    tiles = meta[0:1]
    if recompute:
        _, gate, up = native.gemm_swiglu(x_perm, w1, w3, tile_expert, tiles, save_gate_up=True, align256=True)
    else:
        gate, up = saved[8:10]
    dweights = torch.empty(tokens, 2, dtype=torch.float32, device=dout.device)   # every slot has its row
    dy_perm = native.moe_gather(dout, row_slot, meta, cap, scale=weights.view(-1), y_perm=y_perm,
                                dweights=dweights.view(-1))
    dgu, h = native.gemm_nn_swiglu_bwd(dy_perm, w2, gate, up, tile_expert=tile_expert, num_m_tiles=tiles,
                                       num_experts=experts, align256=True, live_rows=meta[1:2])
    del gate, up
    dx_perm = native.gemm_nn(dgu, w1, w2=w3, tile_expert=tile_expert, num_m_tiles=tiles, num_experts=experts,
                             align256=True)
    # the reduction stops at each expert's own rows: its padding rows are zeros
    dw2 = _wgrad(dy_perm, h, w2, offs, experts, counts)
    dw1, dw3 = _wgrad_gate_up(dgu, x_perm, w1, w3, offs, experts, counts)
    return dx_perm, dweights, dw1, dw2, dw3


class _MoEFused(torch.autograd.Function):
    """The experts for given routing weights, when the expert group is this rank alone."""

    @staticmethod
    def forward(ctx, x, weights, idx, w1, w2, w3, recompute, budget, wants_grad):
        x = x.contiguous()
        weights = weights.float().contiguous()
        out, ctx.recompute, ctx.ledger, saved = _experts_forward(x, weights, idx, w1, w2, w3, recompute, budget,
                                                                 wants_grad)
        ctx.params, ctx.budget = (w1, w2, w3), budget
        ctx.save_for_backward(*saved)
        return out

    @staticmethod
    def backward(ctx, dout):
        *saved, counts = ctx.saved_tensors
        dx_perm, dweights, dw1, dw2, dw3 = _experts_backward(dout.contiguous(), saved, counts, *ctx.params, ctx.recompute)
        dx = native.moe_combine(dx_perm, saved[6], None, dweights.shape[0])
        if ctx.ledger is not None:
            ctx.budget.leave(*ctx.ledger)
        return dx, dweights, None, dw1, dw2, dw3, None, None, None


class _MoELayer(torch.autograd.Function):
    """Router and experts of one rank as one node: the router's product, softmax and choice are one launch, and so are
    its backward, its share of ``dx``, the combine of the expert rows and the sum of both.  ``residual``, if given, is
    added by the forward combine.  With ``balance`` the balance loss is a second output, one kernel over the router's
    probabilities; its gradient joins the router's in the ``dx`` kernel."""

    @staticmethod
    def forward(ctx, x, router_w, w1, w2, w3, residual, recompute, budget, balance, wants_grad):
        ctx.set_materialize_grads(False)
        weights, idx, probs = native.router_fwd(x, router_w)
        out, ctx.recompute, ctx.ledger, saved = _experts_forward(x, weights, idx, w1, w2, w3, recompute, budget,
                                                                 wants_grad, residual)
        ctx.params, ctx.router_w, ctx.budget = (w1, w2, w3), router_w, budget
        counts = saved.pop()
        ctx.save_for_backward(x, probs, idx, counts, *saved)
        return (out, native.moe_aux(probs, counts)) if balance else out

    @staticmethod
    def backward(ctx, dout, daux=None):
        x, probs, idx, counts, *saved = ctx.saved_tensors
        router_w = ctx.router_w
        dresidual = dout if ctx.needs_input_grad[5] else None
        if dout is None:
            dout = torch.zeros_like(x)
        if daux is not None:
            daux = daux.to(device=x.device, dtype=torch.float32)
        dx_perm, dweights, dw1, dw2, dw3 = _experts_backward(dout.contiguous(), saved, counts, *ctx.params, ctx.recompute)
        dx, dlogits = native.moe_dx(dx_perm, saved[6], dweights, probs, idx, saved[2], router_w, daux,
                                    counts)
        main_grad = getattr(router_w, "main_grad", None)
        drouter = None
        if main_grad is not None:
            native.gemm_tn(dlogits, x, out=main_grad, accumulate=True)
        elif ctx.needs_input_grad[1]:
            drouter = native.gemm_tn(dlogits, x, out_dtype=router_w.dtype)
        if ctx.ledger is not None:
            ctx.budget.leave(*ctx.ledger)
        return dx, drouter, dw1, dw2, dw3, dresidual, None, None, None, None


def moe_layer_node(x, router_w, w1, w2, w3, residual=None, recompute: bool = False, balance: bool = False):
    """The routed layer of ``x [..., D]`` as a C++ node (``csrc/nodes.cpp: MoELayer``; the steps of ``_MoELayer``, which
    stays for callers with an activation budget, for weights without gradient buffers and for what the node does not take):
    its output, with ``balance`` and its balance loss, or ``None``."""
    grouter = getattr(router_w, "main_grad", None)
    g1, g3, g2 = getattr(w1, "main_grad", None), getattr(w3, "main_grad", None), getattr(w2, "main_grad", None)
    if (grouter is None or g1 is None or g2 is None or g3 is None or getattr(router_w, "pending_gather", None) is not None):
        return None
    nodes = cpp_nodes(x, router_w, w1, w3, w2, grouter, g1, g3, g2, *(() if residual is None else (residual,)))
    done = nodes.moe_layer(x, router_w, w1, w3, w2, residual, grouter, g1, g3, g2, native.status_word(x.device), ALIGN,
                           recompute, balance) if nodes else None
    return done if balance or done is None else done[0]


def moe_layer_fused(x, router_w, w1, w2, w3, residual=None, recompute: bool = False, budget=None,
                    balance: bool = False):
    """Output of a routed layer on one rank (with ``balance``: and its balance loss), or ``None`` where the router has
    to run by itself: more than 16 experts (or more router weights than a CTA stages), a weight that is still to be
    gathered, layouts that the 16-byte accesses do not take."""
    experts, dim = router_w.shape
    if not (2 <= experts <= 16 and experts == w1.shape[0] and dim == x.shape[1] and dim % 8 == 0
            and experts * dim * 2 <= 200 * 1024 and x.shape[0] > 0
            and getattr(router_w, "pending_gather", None) is None
            and all(t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0
                    for t in ((x, router_w) if residual is None else (x, router_w, residual)))):
        return None
    return _MoELayer.apply(x, router_w, w1, w2, w3, residual, recompute, budget, balance,
                           backward_follows(x, router_w, w1, w2, w3, residual))


def moe_ffn_fused(x, weights, idx, w1, w2, w3, recompute: bool = False, budget=None):
    """The block on one rank.  ``budget`` (``parallel.memory.ActivationBudget``): when given, the call keeps its
    gate/up pre-activations only while the budget has room and rebuilds them in the backward pass otherwise."""
    return _MoEFused.apply(x, weights, idx, w1, w2, w3, recompute, budget, backward_follows(x, weights, w1, w2, w3))


# ----------------------------------------------------------------------------- expert-parallel path (comm/ep.py)
class _StageIn(torch.autograd.Function):
    """Copy the block input into a pool slot that the other ranks of the expert group can read.  The router and
    the MoE op both consume the slot tensor, so this node's backward runs after theirs and gives the slot back."""

    @staticmethod
    def forward(ctx, x, epc, slot):
        ctx.epc, ctx.slot = epc, slot
        staged = epc.slot_tensor(slot)
        staged.copy_(x)
        return staged.view_as(x)

    @staticmethod
    def backward(ctx, dx):
        ctx.epc.release(ctx.slot)
        return dx, None, None


class _MoEPull(torch.autograd.Function):
    """The MoE block on ``comm.ep.EPPull``: plan -> gather+gate/up+SwiGLU (one kernel) -> down projection with the
    weighted return in its epilogue -> combine.  Backward: gather+dh (one kernel), gather x again and rebuild the
    gate/up rows that were not kept (one kernel), SwiGLU backward, dx with the return in its epilogue, the three
    weight-gradient GEMMs, combine."""

    @staticmethod
    def forward(ctx, x, weights, idx, w1, w2, w3, recompute, epc, key, budget, slot, wants_grad):
        from ..comm import ep as E
        g = epc.g
        tokens, dim = x.shape
        ffn = w1.shape[1]
        weights = weights.float().contiguous()
        offs, seg_live_end, tile_expert, meta, seq = epc.plan(idx, weights, key)
        cap_saved, ledger = 0, None
        if wants_grad and not recompute:
            cap_saved = epc.expected_rows(key)
            if budget is not None:
                ledger = (0, cap_saved * ffn * 4)
                kept = budget.enter(*ledger)
                ledger += (kept,)
                if not kept:
                    cap_saved = 0
        dev = x.device
        gate = torch.empty(cap_saved, ffn, dtype=torch.bfloat16, device=dev) if cap_saved else None
        up = torch.empty(cap_saved, ffn, dtype=torch.bfloat16, device=dev) if cap_saved else None
        row_src = torch.empty(epc.cap, dtype=torch.int32, device=dev)
        row_tag = torch.empty(epc.cap, dtype=torch.int32, device=dev)
        row_w = torch.empty(epc.cap, dtype=torch.float32, device=dev)
        x_ws, h = epc.ws("x", dim), epc.ws("h", ffn)
        epc.gather_gemm(0, x_ws, w1, w3, 2 * ffn, dim, tile_expert, meta, seg_live_end, 0, epc.pool[slot].table(), 1,
                        epc.land_src.tensor, epc.land_tag.tensor, epc.land_w.tensor, (row_src, row_tag, row_w),
                        E.SIG_META, seq, 1, h, gate, up, None, None, cap_saved)
        ret_seq = g.next_seq(E.SIG_RET_F)
        native.gemm_nt_push(h, w2, tile_expert, meta[0:1], epc.e_local, epc.ret_f.table(), row_tag, row_src, row_w,
                            g.sig.table(), E.SIG_RET_F, ret_seq, g.rank, epc.ep, epc.tickets[4:])
        out, _ = epc.combine(epc.ret_f, E.SIG_RET_F, ret_seq, with_scalars=False)
        ctx.params = (w1, w2, w3)
        ctx.meta_py = (tokens, dim, ffn, epc, slot, cap_saved)
        ctx.budget, ctx.ledger = budget, ledger
        saved = [offs, seg_live_end, tile_expert, meta, row_src, row_tag, row_w]
        if cap_saved:
            saved += [gate, up]
        ctx.save_for_backward(*saved)
        return out

    @staticmethod
    def backward(ctx, dout):
        from ..comm import ep as E
        w1, w2, w3 = ctx.params
        tokens, dim, ffn, epc, slot, cap_saved = ctx.meta_py
        saved = list(ctx.saved_tensors)
        offs, seg_live_end, tile_expert, meta, row_src, row_tag, row_w = saved[:7]
        gate, up = saved[7:9] if cap_saved else (None, None)
        g = epc.g
        experts = epc.e_local
        tiles = meta[0:1]
        epc.dout.tensor.view(tokens, dim).copy_(dout)
        dy_ws, x_ws, dh, dgu = epc.ws("dy", dim), epc.ws("x", dim), epc.ws("h", ffn), epc.ws("dgu", 2 * ffn)
        gate_ws, up_ws = epc.ws("gate", ffn), epc.ws("up", ffn)
        # dh = dy_perm W2, the rows of dy fetched from the peers' staged output gradients by the same kernel
        bseq = g.next_seq(E.SIG_BDATA)
        epc.gather_gemm(1, dy_ws, w2, None, ffn, dim, tile_expert, meta, seg_live_end, 0, epc.dout.table(), 1,
                        row_src, row_tag, None, None, E.SIG_BDATA, bseq, 2, dh, None, None, None, None, 0)
        # x rows again (for the weight gradients), gate/up rebuilt for the rows that were not kept
        epc.gather_gemm(0, x_ws, w1, w3, 2 * ffn, dim, tile_expert, meta, seg_live_end, cap_saved // 128,
                        epc.pool[slot].table(), 1, row_src, row_tag, None, None, 0, 0, 0, None, None, None, gate_ws,
                        up_ws, cap_saved)
        native.ep_swiglu_bwd(dh, gate, up, gate_ws, up_ws, cap_saved, dgu, meta, row_tag, row_src, row_w,
                             epc.dw_ret.table(), epc.ep)
        ret_seq = g.next_seq(E.SIG_RET_B)
        native.gemm_nn_push(dgu, w1, w3, tile_expert, tiles, experts, epc.ret_b.table(), row_tag, row_src, None,
                            g.sig.table(), E.SIG_RET_B, ret_seq, g.rank, epc.ep, epc.tickets[5:])
        dw2 = _wgrad(dy_ws, dh, w2, offs, experts)
        dw1 = _wgrad(dgu[:, :ffn], x_ws, w1, offs, experts)
        dw3 = _wgrad(dgu[:, ffn:], x_ws, w3, offs, experts)
        dx, dweights = epc.combine(epc.ret_b, E.SIG_RET_B, ret_seq, with_scalars=True)
        if ctx.ledger is not None:
            ctx.budget.leave(*ctx.ledger)
        return dx, dweights, None, dw1, dw2, dw3, None, None, None, None, None, None


def moe_ffn_pull(x, weights_of, w1, w2, w3, epc, recompute: bool = False, key=None, budget=None):
    """MoE block over the expert group of ``epc`` (``comm.ep.EPPull``).  ``weights_of(staged)`` computes the router's
    ``(weights, idx)`` from the staged copy of ``x`` (so that the router keeps the pool slot, not a second copy of
    the activations, for its backward pass)."""
    slot = epc.acquire()
    staged = _StageIn.apply(x.contiguous(), epc, slot)
    weights, idx = weights_of(staged)
    out = _MoEPull.apply(staged, weights, idx, w1, w2, w3, recompute, epc, key if key is not None else id(w1), budget,
                         slot, backward_follows(staged, weights, w1, w2, w3))
    if not (torch.is_grad_enabled() and (x.requires_grad or weights.requires_grad)):
        epc.release(slot)          # no backward pass will come for this call
    return out, weights, idx
