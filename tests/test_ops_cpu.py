"""PyTorch statements of the ops against independent formulations."""
import math

import pytest
import torch
import torch.nn.functional as F

from b200moe import ops
from b200moe.ops import functional as Fn
from b200moe.ops.moe import build_plan, grouped_swiglu
from b200moe.optim import AdamW
from b200moe.utils.schedule import learning_rate_schedule_wrapper


def test_softmax_silu_cross_entropy_match_torch():
    x = torch.randn(5, 11)
    assert torch.allclose(Fn.softmax(x, -1), torch.softmax(x, -1), atol=1e-6)
    assert torch.allclose(Fn.log_softmax(x), torch.log_softmax(x, -1), atol=1e-6)
    assert torch.allclose(Fn.silu(x), F.silu(x), atol=1e-6)
    t = torch.randint(0, 11, (5,))
    assert torch.allclose(Fn.cross_entropy(x, t), F.cross_entropy(x, t), atol=1e-6)
    mask = (torch.rand(5, 11) > 0.3).float()
    mask[:, 0] = 1
    want = torch.softmax(x.masked_fill(mask == 0, float("-inf")), -1)
    assert torch.allclose(Fn.softmax(x, -1, mask), want, atol=1e-6)


def test_rmsnorm_and_fused_add():
    x, d, w = torch.randn(3, 7, 16), torch.randn(3, 7, 16), torch.rand(16) + 0.5
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w
    assert torch.allclose(ops.rmsnorm(x, w), want, atol=1e-5)
    s, y = ops.add_rmsnorm(x, d, w)
    assert torch.allclose(s, x + d) and torch.allclose(y, Fn.rmsnorm_ref(x + d, w), atol=1e-6)


def test_rope_is_pairwise_rotation_with_reference_frequencies():
    hd, seq, theta = 8, 6, 10000.0
    cos, sin = Fn.rope_tables(theta, hd, seq)
    x = torch.randn(2, 3, seq, hd)
    out = Fn.apply_rope_ref(x, cos, sin)
    for pos in range(seq):
        for i in range(hd // 2):
            angle = pos * theta ** ((2 - 2 * (i + 1)) / hd)
            a, b = x[..., pos, 2 * i], x[..., pos, 2 * i + 1]
            assert torch.allclose(out[..., pos, 2 * i], a * math.cos(angle) - b * math.sin(angle), atol=1e-5)
            assert torch.allclose(out[..., pos, 2 * i + 1], a * math.sin(angle) + b * math.cos(angle), atol=1e-5)
    assert torch.allclose(out.norm(dim=-1), x.norm(dim=-1), atol=1e-5)


def test_attention_is_causal_gqa():
    B, S, Hq, Hkv, hd = 2, 12, 8, 2, 16
    q, k, v = torch.randn(B, S, Hq, hd), torch.randn(B, S, Hkv, hd), torch.randn(B, S, Hkv, hd)
    out = ops.rope_attention(q, k, v, None, None)
    scores = torch.einsum("bshd,bthd->bhst", q, k.repeat_interleave(4, 2)) / math.sqrt(hd)
    scores = scores.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool), 1), float("-inf"))
    want = torch.einsum("bhst,bthd->bshd", scores.softmax(-1), v.repeat_interleave(4, 2))
    assert torch.allclose(out, want, atol=1e-5)


def test_router_top2_renormalises():
    logits = torch.randn(64, 8)
    w, idx = ops.router_top2(logits)
    p = logits.softmax(-1)
    top, ti = p.topk(2, -1)
    assert torch.equal(idx, ti)
    assert torch.allclose(w, top / top.sum(-1, keepdim=True), atol=1e-6)
    assert torch.allclose(w.sum(-1), torch.ones(64), atol=1e-6)


@pytest.mark.parametrize("pattern", ["random", "one_expert", "empty_experts"])
def test_plan_layout_and_padding(pattern):
    T, E = 50, 4
    if pattern == "random":
        idx = torch.stack([torch.randperm(E)[:2] for _ in range(T)])
    elif pattern == "one_expert":
        idx = torch.tensor([[2, 0]] * T)
    else:
        idx = torch.tensor([[1, 3]] * T)
    plan = build_plan(idx, E, None, align=16)
    flat = idx.reshape(-1)
    assert torch.equal(flat[plan.order], flat.sort(stable=True).values)
    ends = plan.offs.tolist()
    assert all(e % 16 == 0 for e in ends) and ends[-1] <= plan.rows
    start = 0
    sorted_experts = flat[plan.order]
    for e, end in enumerate(ends):
        rows = plan.recv_to_row[sorted_experts == e]
        n = int((flat == e).sum())
        assert rows.numel() == n
        if n:
            assert torch.equal(rows, torch.arange(start, start + n))
        assert end - start >= n and end - start < n + 16
        start = end


def test_grouped_swiglu_backward_matches_autograd():
    torch.manual_seed(0)
    E, D, Fd, rows = 3, 8, 12, 48
    offs = torch.tensor([16, 16, 48], dtype=torch.int32)
    x = torch.randn(rows, D, requires_grad=True)
    w1, w2, w3 = (torch.randn(E, Fd, D, requires_grad=True), torch.randn(E, D, Fd, requires_grad=True),
                  torch.randn(E, Fd, D, requires_grad=True))
    dy = torch.randn(rows, D)
    for recompute in (False, True):
        for t in (x, w1, w2, w3):
            t.grad = None
        grouped_swiglu(x, w1, w2, w3, offs, recompute).backward(dy)
        got = [t.grad.clone() for t in (x, w1, w2, w3)]
        for t in (x, w1, w2, w3):
            t.grad = None
        y, start = torch.zeros(rows, D), 0
        parts = []
        for e, end in enumerate(offs.tolist()):
            xe = x[start:end]
            parts.append((F.silu(xe @ w1[e].T) * (xe @ w3[e].T)) @ w2[e].T)
            start = end
        torch.cat(parts).backward(dy)
        for g, t in zip(got, (x, w1, w2, w3)):
            assert torch.allclose(g, t.grad, atol=1e-4, rtol=1e-4)


def test_linear_accumulates_into_main_grad():
    w = torch.randn(6, 4, requires_grad=True)
    w.main_grad = torch.zeros(6, 4)
    x = torch.randn(5, 4, requires_grad=True)
    dy = torch.randn(5, 6)
    for _ in range(2):
        ops.linear(x, w).backward(dy)
    assert w.grad is None
    assert torch.allclose(w.main_grad, 2 * dy.T @ x.detach(), atol=1e-5)
    assert torch.allclose(x.grad, 2 * dy @ w.detach(), atol=1e-5)


def test_lm_head_cross_entropy_equals_two_step():
    h, w = torch.randn(2, 5, 8, requires_grad=True), torch.randn(20, 8, requires_grad=True)
    t = torch.randint(0, 20, (2, 5))
    a = ops.lm_head_cross_entropy(h, w, t)
    b = F.cross_entropy((h @ w.T).reshape(-1, 20), t.reshape(-1))
    assert torch.allclose(a, b, atol=1e-6)


def test_lr_schedule_shape():
    f = learning_rate_schedule_wrapper(1.0, 0.1, 10, 110)
    assert f(0) == 0 and f(5) == 0.5 and abs(f(10) - 1.0) < 1e-12
    assert abs(f(60) - 0.55) < 1e-12 and abs(f(110) - 0.1) < 1e-12 and f(500) == 0.1


@pytest.mark.parametrize("state_dtype", [torch.float32, torch.bfloat16])
def test_adamw_matches_closed_form(state_dtype):
    torch.manual_seed(0)
    p = torch.nn.Parameter(torch.randn(7, 3))
    ref = p.detach().clone()
    opt = AdamW([p], lr=1e-2, betas=(0.9, 0.99), eps=1e-8, weight_decay=0.1, state_dtype=state_dtype)
    m = torch.zeros_like(ref)
    v = torch.zeros_like(ref)
    for t in range(1, 4):
        g = torch.randn(7, 3)
        p.grad = g.clone()
        opt.step()
        ref = ref * (1 - 1e-2 * 0.1)
        m = 0.9 * m + 0.1 * g
        v = 0.99 * v + 0.01 * g * g
        ref = ref - 1e-2 * math.sqrt(1 - 0.99 ** t) / (1 - 0.9 ** t) * m / (v.sqrt() + 1e-8)
        if state_dtype == torch.bfloat16:
            m, v = m.bfloat16().float(), v.bfloat16().float()
    tol = 1e-6 if state_dtype == torch.float32 else 2e-3
    assert torch.allclose(p.detach(), ref, atol=tol)
    assert opt.param_groups[0]["t"] == 4
    sd = opt.state_dict()
    assert set(sd["state"][0]) == {"m", "v"}
    assert {"lr", "beta1", "beta2", "t", "epsilon", "lambda_"} <= set(sd["param_groups"][0])


def test_gradient_clipping_and_sampler():
    ps = [torch.nn.Parameter(torch.ones(4)), torch.nn.Parameter(torch.ones(3))]
    for p in ps:
        p.grad = torch.full_like(p, 2.0)
    norm = Fn.gradient_clipping(ps, 1.0)
    assert abs(float(norm) - math.sqrt(28)) < 1e-5
    total = math.sqrt(sum(float((p.grad ** 2).sum()) for p in ps))
    assert abs(total - 1.0) < 1e-4
    logits = torch.tensor([[0.0, 10.0, 0.0]])
    assert int(Fn.sample_output(logits, t=1.0, p=0.0)) == 1


def test_linear_consumes_a_pending_gather_once():
    """A weight may carry the call that gathers its peer rows and multiplies (all-gather fused with the GEMM);
    the first ``linear`` after an optimizer step uses it, later ones and the backward pass use the weight."""
    import torch
    from b200moe import ops
    torch.manual_seed(0)
    x = torch.randn(6, 8, requires_grad=True)
    w = torch.randn(5, 8, requires_grad=True)
    calls = []

    def gather(x2d):
        calls.append(tuple(x2d.shape))
        return x2d.detach() @ w.detach().t()

    w.pending_gather = gather
    y = ops.linear(x, w)
    assert calls == [(6, 8)] and w.pending_gather is None
    assert torch.allclose(y, x @ w.t(), atol=1e-6)
    y.sum().backward()
    assert torch.allclose(x.grad, torch.ones(6, 5) @ w.detach(), atol=1e-6)
    assert torch.allclose(w.grad, torch.ones(6, 5).t() @ x.detach(), atol=1e-6)
    ops.linear(x, w)
    assert calls == [(6, 8)]


def test_fsdp_first_use_gather_needs_the_fused_backend():
    """On CPU (no peer-memory backend) ``gather="first_use"`` marks nothing lazy and training is unchanged."""
    import torch
    from b200moe.models import TransformerLMPipelined
    from b200moe.parallel import FSDPWrapperPipelined
    torch.manual_seed(0)
    model = TransformerLMPipelined(64, 32, 32, 1, 4, 0, 1, num_expert_per_node=2, d_ff=64)
    wrapped = FSDPWrapperPipelined(model, None, None, compute_dtype=torch.float32, gather="first_use")
    assert wrapped._lazy == [] and not any(e.get("lazy") for e in wrapped.flat.entries)
    with pytest.raises(ValueError):
        FSDPWrapperPipelined(model, None, None, gather="sometimes")


def test_rotary_tables_that_the_kernels_would_read_past_are_refused(monkeypatch):
    """Refused before anything is launched: tables shorter than the sequence or of a narrower type.  A table that
    starts off a 16-byte boundary is copied."""
    from b200moe.ops import native
    launched = []
    monkeypatch.setattr(native, "_call", lambda name, *args, **kw: launched.append((name, args)))
    monkeypatch.setattr(native, "_stream", lambda: None)
    S, hd = 130, 128
    cos, sin = Fn.rope_tables(10000.0, hd, S)
    q, k = torch.zeros(1, S, 4, hd, dtype=torch.bfloat16), torch.zeros(1, S, 1, hd, dtype=torch.bfloat16)
    for bad in (cos[:S - 1], cos.bfloat16()):
        for pair in ((bad, sin), (cos, bad)):
            with pytest.raises(ValueError):
                native.attention_fwd(q, k, k, *pair)
            with pytest.raises(ValueError):
                native.rope_inplace(q, 0, S, S, 4, hd, 4 * hd, *pair, 1.0)
    assert launched == []
    shifted = torch.cat((torch.zeros(1), cos.reshape(-1)))[1:].view(S, -1)
    native.rope_inplace(q, 0, S, S, 4, hd, 4 * hd, shifted, sin, 1.0)
    (name, args), = launched
    assert name == "b2_rope" and args[1].value % 16 == 0 and args[1].value != shifted.data_ptr()
    assert args[2].value == sin.data_ptr()


def test_dense_swiglu_keeps_gate_and_up_only_where_a_backward_pass_can_follow(monkeypatch):
    from b200moe.ops import dense, native
    kept = []

    def gemm_swiglu(x, w1, w3, save_gate_up=True):
        kept.append(save_gate_up)
        return (x.new_zeros(x.shape[0], w1.shape[1]),) * 3

    monkeypatch.setattr(dense, "use_native", lambda *_: True)
    monkeypatch.setattr(native, "gemm_swiglu", gemm_swiglu)
    monkeypatch.setattr(native, "gemm_nt", lambda x, w: x.new_zeros(x.shape[0], w.shape[0]))
    x = torch.zeros(3, 64, dtype=torch.bfloat16)
    weights = [torch.zeros(s, dtype=torch.bfloat16, requires_grad=True) for s in ((128, 64), (128, 64), (64, 128))]
    assert ops.swiglu_ffn(x, *weights).requires_grad
    with torch.no_grad():
        ops.swiglu_ffn(x, *weights)
    assert not ops.swiglu_ffn(x, *(w.detach() for w in weights)).requires_grad
    assert kept == [True, False, False]


@pytest.mark.parametrize("form", ["layer", "experts"])
def test_routed_experts_charge_the_budget_only_where_a_backward_pass_can_follow(monkeypatch, form):
    """Evaluation and the first forward pass of a recomputed block keep no gate and up, and leave the activation budget
    as it was: no backward pass comes that would give the charge back."""
    from b200moe.ops import moe_fused, native
    from b200moe.parallel.memory import ActivationBudget
    T, D, F, E = 5, 8, 16, 2
    kept = []

    def gemm_swiglu(x, w1, w3, tile_expert, tiles, save_gate_up, align256):
        kept.append(save_gate_up)
        return x.new_zeros(x.shape[0], F), x.new_zeros(1), x.new_zeros(1)

    table = torch.zeros(4, dtype=torch.int32)
    monkeypatch.setattr(native, "router_fwd", lambda x, w: (torch.ones(T, 2), torch.zeros(T, 2), torch.ones(T, E)))
    monkeypatch.setattr(native, "moe_plan", lambda *_: (table,) * 6)
    monkeypatch.setattr(native, "moe_gather", lambda x, row_slot, meta, cap: x.new_zeros(cap, D))
    monkeypatch.setattr(native, "gemm_swiglu", gemm_swiglu)
    monkeypatch.setattr(native, "gemm_nt", lambda h, w, **_: h.new_zeros(h.shape[0], D))
    monkeypatch.setattr(native, "moe_combine", lambda y, slot_row, w, tokens, residual=None: y.new_zeros(tokens, D))
    budget = ActivationBudget(1 << 30)
    x = torch.zeros(T, D, dtype=torch.bfloat16)
    w1, w3, w2, router = (torch.zeros(s, dtype=torch.bfloat16, requires_grad=True)
                          for s in ((E, F, D), (E, F, D), (E, D, F), (E, D)))

    def call():
        if form == "layer":
            return moe_fused.moe_layer_fused(x, router, w1, w2, w3, budget=budget)
        return moe_fused.moe_ffn_fused(x, torch.ones(T, 2), torch.zeros(T, 2), w1, w2, w3, budget=budget)

    with torch.no_grad():
        call()
    assert (budget.used, budget.live_calls, budget.granted, budget.refused) == (0, 0, 0, 0)
    assert call().requires_grad
    assert budget.live_calls == 1 and budget.used > 0
    assert kept == [False, True]


def test_head_keeps_whole_logits_only_where_a_backward_pass_can_follow(monkeypatch):
    from b200moe.ops import loss, native
    rows = []

    def gemm_nt(h, w):
        rows.append(h.shape[0])
        return h.new_zeros(h.shape[0], w.shape[0])

    monkeypatch.setattr(loss, "use_native", lambda *_: True)
    monkeypatch.setattr(loss, "CHUNK_TOKENS", 4)
    monkeypatch.setattr(native, "gemm_nt", gemm_nt)
    monkeypatch.setattr(native, "cross_entropy_scaled_", lambda *_: None)
    hidden, targets = torch.zeros(10, 8), torch.zeros(10, dtype=torch.long)
    weight = torch.zeros(16, 8, requires_grad=True)
    with torch.no_grad():
        ops.lm_head_cross_entropy(hidden, weight, targets)
    assert rows == [4, 4, 2]
    rows.clear()
    assert ops.lm_head_cross_entropy(hidden, weight, targets).requires_grad
    assert rows == [10]


@pytest.mark.parametrize("disabled", ["", "moe", "router", "gemm", "swiglu"])
def test_switching_off_an_op_family_leaves_the_fused_layers_that_replace_it(monkeypatch, disabled):
    from b200moe.models.layers import MoELayerMulti
    from b200moe.ops import dense, moe_fused
    monkeypatch.setattr(ops, "use_native", lambda t, op="": op != disabled)
    monkeypatch.setattr(dense, "use_native", lambda t, op="": op != disabled)
    monkeypatch.setattr(moe_fused, "moe_layer_fused", lambda *_, **__: "fused")
    monkeypatch.setattr(dense._SwiGLUFFN, "apply", lambda *_: "fused")
    layer = MoELayerMulti(64, 128, num_expert_per_node=2)
    x = torch.zeros(3, 64, dtype=torch.bfloat16)
    assert (layer._fused(x, None, False) is None) == (disabled in ("moe", "router", "gemm"))
    weights = [torch.zeros(s, dtype=torch.bfloat16) for s in ((128, 64), (128, 64), (64, 128))]
    assert (ops.swiglu_ffn(x, *weights) is None) == (disabled in ("gemm", "swiglu"))


def test_differentiable_attention_refuses_fp16_before_it_runs(monkeypatch):
    """The fp16 kernel has no backward pass: an error in the forward call, not later."""
    from b200moe.ops import attention, native
    monkeypatch.setattr(attention, "use_native", lambda *_: True)
    monkeypatch.setattr(native, "attention_fwd", lambda q, k, v, cos, sin: (q, q.new_zeros(1), q, k))
    q = torch.zeros(1, 128, 1, 128, dtype=torch.float16, requires_grad=True)
    with pytest.raises(TypeError):
        ops.rope_attention(q, q, q, None, None)
    q = torch.zeros(1, 128, 1, 128, dtype=torch.bfloat16, requires_grad=True)
    assert ops.rope_attention(q, q, q, None, None).requires_grad


def test_adamw_zero_grad_is_seen_by_a_profiler():
    p = torch.nn.Parameter(torch.ones(3))
    optimizer = AdamW([p])
    for profiled in (True, False):
        p.grad = torch.ones(3)
        if profiled:
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as seen:
                optimizer.zero_grad()
            assert "Optimizer.zero_grad#AdamW.zero_grad" in [event.key for event in seen.key_averages()]
        else:
            optimizer.zero_grad()
        assert p.grad is None
