"""Performance cases of the framework on one GPU: what a training or evaluation program has it do, through the public
entry points that such a program calls.

Kinds of case (a case is a dict of plain values; ``kind`` selects the path):

``step``      one optimizer step of the decoder: ``pipelined_train_overlap`` on a wrapped model, all microbatches,
              gradient accumulation, AdamW, refreshed compute weights
``logits``    evaluation: logits of a batch of prompts, no gradients
``moe``       one expert layer (router, dispatch, experts, combine), forward and backward
``ffn``       a dense SwiGLU stack, forward and backward (the module microbenchmark's module)
``rope_attn`` causal grouped-query attention with rotary embedding, forward and backward
``attn``      attention without rotation, causal or not, forward and backward
``flash``     the forward-only ``[B, H, S, 128]`` attention entry point (fp16 or bf16, not causal)
``head``      LM head with cross-entropy, forward and backward
``adamw``     one optimizer update of dense fp32 and expert bf16 parameters

Inputs are made on the GPU from the seed alone: uniform token ids, unit-variance activations, the layers' own
initialisers for weights.
"""
import math

import torch

from b200moe import ops
from b200moe.models import TransformerLMPipelined
from b200moe.models.layers import MoELayerMulti
from b200moe.models.module_dev import ModuleStack
from b200moe.ops.attention import attention, flash_attention_forward
from b200moe.ops.functional import cross_entropy, rope_tables
from b200moe.optim import AdamW
from b200moe.parallel import FSDPWrapperPipelined, pipelined_train_overlap

BF16 = torch.bfloat16
HEAD_DIM = 128


def listed():
    return [
        # the small decoder of the smoke run: two narrow blocks, 2 microbatches of 2 x 512 tokens; a step is hundreds of
        # short launches, so host time and launch gaps count
        {"name": "step_small", "kind": "step", "d_model": 512, "heads": 4, "blocks": 2, "experts": 4, "d_ff": 1024,
         "vocab": 2048, "seq": 512, "batch": 4, "microbatches": 2, "aux": 0.0, "expert_state": "float32"},
        # a research-size decoder (width 1024, d_ff = 3.5 width as in the 8x7B-like configuration), sequence 1024, with
        # the router's auxiliary loss switched on
        {"name": "step_medium", "kind": "step", "d_model": 1024, "heads": 8, "blocks": 4, "experts": 8, "d_ff": 3584,
         "vocab": 32000, "seq": 1024, "batch": 8, "microbatches": 2, "aux": 0.01, "expert_state": "float32"},
        # one block of the headline configuration with its embedding and head: microbatches of 2 x 8192 tokens, expert
        # gradients and moments in bf16 as on one GPU
        {"name": "step_block", "kind": "step", "d_model": 4096, "heads": 32, "blocks": 1, "experts": 8, "d_ff": 14336,
         "vocab": 32000, "seq": 8192, "batch": 4, "microbatches": 2, "aux": 0.0, "expert_state": "bfloat16"},
        # evaluation of three prompts whose length is no multiple of anything
        {"name": "logits_ragged", "kind": "logits", "d_model": 2048, "heads": 16, "blocks": 2, "experts": 8,
         "d_ff": 7168, "vocab": 32000, "seq": 1003, "batch": 3},
        # one expert layer at the widths of the unit tests with a few hundred tokens: the smallest forward/backward call
        {"name": "moe_small", "kind": "moe", "d_model": 512, "d_ff": 1024, "experts": 4, "tokens": 200},
        # one expert layer of the headline configuration on an odd number of tokens (a short, ragged microbatch)
        {"name": "moe_ragged", "kind": "moe", "d_model": 4096, "d_ff": 14336, "experts": 8, "tokens": 5003},
        # the module microbenchmark of the run configuration: three dense SwiGLU layers on [1, 4096, 4096]
        {"name": "ffn_stack", "kind": "ffn", "d_model": 4096, "d_ff": 14336, "batch": 1, "seq": 4096},
        # attention of one headline sequence: 32 query heads, 8 KV heads, 8192 tokens
        {"name": "attn_long", "kind": "rope_attn", "batch": 1, "seq": 8192, "heads": 32, "kv_heads": 8},
        # many short sequences, every query sees every key, as many KV heads as query heads
        {"name": "attn_full_short", "kind": "attn", "batch": 8, "seq": 640, "heads": 16, "kv_heads": 16,
         "causal": False},
        # the stand-alone forward kernel's entry point, fp16
        {"name": "flash_fp16", "kind": "flash", "batch": 2, "heads": 16, "seq": 2048, "dtype": "float16"},
        # LM head and loss of an odd number of tokens
        {"name": "head_loss", "kind": "head", "d_model": 2048, "vocab": 32000, "tokens": 6001},
        # optimizer update of one block with four experts: fp32 dense parameters, bf16 experts with bf16 moments
        {"name": "adamw_block", "kind": "adamw", "d_model": 4096, "d_ff": 14336, "experts": 4,
         "expert_state": "bfloat16"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _sequence(rng, low, high):
    """A sequence length: two in three are multiples of 128, the others are whatever comes."""
    value = _log_int(rng, low, high)
    return max(128, value // 128 * 128) if rng.random() < 0.67 else value


def draw(rng):
    kind = rng.choice(["step", "step", "logits", "moe", "moe", "ffn", "rope_attn", "attn", "flash", "head", "adamw"])
    width = rng.choice([512, 1024, 2048])
    if kind == "step":
        seq = _sequence(rng, 128, 2048)
        microbatches = rng.choice([1, 2, 4])
        return {"kind": kind, "d_model": width, "heads": width // HEAD_DIM, "blocks": rng.choice([1, 2, 3, 4]),
                "experts": rng.choice([4, 8]), "d_ff": width * 7 // 2, "vocab": rng.choice([2048, 32000]), "seq": seq,
                "batch": microbatches * _log_int(rng, 1, 8), "microbatches": microbatches,
                "aux": rng.choice([0.0, 0.01]), "expert_state": rng.choice(["float32", "bfloat16"])}
    if kind == "logits":
        return {"kind": kind, "d_model": width, "heads": width // HEAD_DIM, "blocks": rng.choice([1, 2]),
                "experts": rng.choice([4, 8]), "d_ff": width * 7 // 2, "vocab": 32000,
                "seq": _sequence(rng, 64, 4096), "batch": rng.choice([1, 2, 3, 4])}
    if kind == "moe":
        width = rng.choice([512, 1024, 2048, 4096])
        return {"kind": kind, "d_model": width, "d_ff": width * 7 // 2, "experts": rng.choice([4, 8]),
                "tokens": _log_int(rng, 100, 16384)}
    if kind == "ffn":
        width = rng.choice([1024, 2048, 4096])
        return {"kind": kind, "d_model": width, "d_ff": width * 7 // 2, "batch": rng.choice([1, 2, 4]),
                "seq": _log_int(rng, 64, 4096)}
    if kind == "rope_attn":
        heads = rng.choice([8, 16, 32])
        return {"kind": kind, "batch": rng.choice([1, 2, 3]), "seq": _sequence(rng, 128, 8192), "heads": heads,
                "kv_heads": heads // 4}
    if kind == "attn":
        heads = rng.choice([4, 8, 16])
        return {"kind": kind, "batch": rng.choice([1, 2, 4, 8]), "seq": _sequence(rng, 128, 4096), "heads": heads,
                "kv_heads": heads // rng.choice([1, 2, 4]), "causal": rng.random() < 0.5}
    if kind == "flash":
        return {"kind": kind, "batch": rng.choice([1, 2, 4]), "heads": rng.choice([4, 8, 16]),
                "seq": max(128, _log_int(rng, 128, 4096) // 128 * 128), "dtype": rng.choice(["float16", "bfloat16"])}
    if kind == "head":
        return {"kind": kind, "d_model": rng.choice([512, 1024, 2048, 4096]), "vocab": 32000,
                "tokens": _log_int(rng, 100, 16384)}
    width = 128 * _log_int(rng, 4, 32)
    return {"kind": kind, "d_model": width, "d_ff": width * 7 // 2, "experts": rng.choice([1, 2, 3, 4]),
            "expert_state": rng.choice(["float32", "bfloat16"])}


# ------------------------------------------------------------------------------ states
def _decoder(case):
    with torch.device("cuda"):
        model = TransformerLMPipelined(case["vocab"], case["seq"], case["d_model"], case["blocks"], case["heads"], 0, 1,
                                       num_expert_per_node=case["experts"], d_ff=case["d_ff"])
    experts = getattr(torch, case.get("expert_state", "float32"))
    return FSDPWrapperPipelined(model, None, None, compute_dtype=BF16, expert_grad_dtype=experts,
                                expert_state_dtype=experts)


def _rand(*shape, dtype=BF16, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(dtype)


def prepare(case, seed):
    torch.manual_seed(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind == "step":
        model = _decoder(case)
        optimizer = AdamW(model.parameters(), lr=3e-4, weight_decay=0.01)
        optimizer.materialize_state()
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), device="cuda")
        state.update(model=model, optimizer=optimizer, x=ids[:, :-1].contiguous(), y=ids[:, 1:].contiguous())
    elif kind == "logits":
        state.update(model=_decoder(case),
                     x=torch.randint(0, case["vocab"], (case["batch"], case["seq"]), device="cuda"))
    elif kind == "moe":
        with torch.device("cuda"):
            layer = MoELayerMulti(case["d_model"], case["d_ff"], num_expert_per_node=case["experts"])
        model = FSDPWrapperPipelined(layer, None, None, compute_dtype=BF16, expert_grad_dtype=BF16,
                                     expert_state_dtype=BF16)
        state.update(model=model, x=_rand(case["tokens"], case["d_model"]).requires_grad_(True),
                     dy=_rand(case["tokens"], case["d_model"]))
    elif kind == "ffn":
        with torch.device("cuda"):
            stack = ModuleStack(case["d_model"], case["d_model"], dtype=BF16, d_ff=case["d_ff"])
        shape = (case["batch"], case["seq"], case["d_model"])
        state.update(model=stack, x=_rand(*shape).requires_grad_(True), dy=_rand(*shape))
    elif kind in ("rope_attn", "attn"):
        B, S, H, Hkv = case["batch"], case["seq"], case["heads"], case["kv_heads"]
        state.update(q=_rand(B, S, H, HEAD_DIM).requires_grad_(True),
                     k=_rand(B, S, Hkv, HEAD_DIM).requires_grad_(True),
                     v=_rand(B, S, Hkv, HEAD_DIM).requires_grad_(True), dy=_rand(B, S, H, HEAD_DIM))
        if kind == "rope_attn":
            state["cos"], state["sin"] = rope_tables(10000.0, HEAD_DIM, S, "cuda")
    elif kind == "flash":
        shape = (case["batch"], case["heads"], case["seq"], HEAD_DIM)
        dtype = getattr(torch, case["dtype"])
        state.update(q=_rand(*shape, dtype=dtype), k=_rand(*shape, dtype=dtype), v=_rand(*shape, dtype=dtype))
    elif kind == "head":
        std = math.sqrt(2.0 / (case["d_model"] + case["vocab"]))
        state.update(hidden=_rand(case["tokens"], case["d_model"]).requires_grad_(True),
                     weight=torch.nn.Parameter(_rand(case["vocab"], case["d_model"], scale=std)),
                     targets=torch.randint(0, case["vocab"], (case["tokens"],), device="cuda"))
    elif kind == "adamw":
        params = []
        for shape, dtype in _adamw_shapes(case):
            p = torch.nn.Parameter(_rand(*shape, dtype=dtype, scale=0.02))
            p.grad = _rand(*shape, dtype=dtype, scale=1e-3)
            if dtype == BF16:
                p._state_dtype = getattr(torch, case["expert_state"])
            params.append(p)
        optimizer = AdamW(params, lr=1e-3, weight_decay=0.01)
        optimizer.materialize_state()
        state.update(params=params, optimizer=optimizer)
    else:
        raise ValueError(kind)
    return state


def _adamw_shapes(case):
    d, f, e = case["d_model"], case["d_ff"], case["experts"]
    dense = [(d,), (d, d), (d // 4, d), (d // 4, d), (d, d), (d,), (8, d), (999, d)]
    return [(s, torch.float32) for s in dense] + [(s, BF16) for s in ((e, f, d), (e, d, f), (e, f, d))]


# ------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        model, optimizer = state["model"], state["optimizer"]
        loss = pipelined_train_overlap(model, optimizer, state["x"], state["y"],
                                       [case["batch"], case["seq"], case["d_model"]], case["microbatches"], 0,
                                       cross_entropy, dtype=BF16, device=state["x"].device,
                                       router_aux_loss_coef=case["aux"])
        return {"loss": loss, "weights": [p.detach() for p in model.parameters()]}
    if kind == "logits":
        with torch.no_grad():
            return state["model"](state["x"])
    if kind == "moe":
        model, x = state["model"], state["x"]
        x.grad = None
        model.clear_grad_accumulators()
        out = model(x)
        out.backward(state["dy"])
        model.reduce_accumulated_gradients()
        return [out.detach(), x.grad, model.module.router.weight.grad] + [p.main_grad for p in model.expert_params]
    if kind == "ffn":
        model, x = state["model"], state["x"]
        x.grad = None
        model.zero_grad(set_to_none=True)
        out = model(x)
        out.backward(state["dy"])
        return [out.detach(), x.grad] + [p.grad for p in model.parameters()]
    if kind in ("rope_attn", "attn"):
        q, k, v = state["q"], state["k"], state["v"]
        if kind == "rope_attn":
            out = ops.rope_attention(q, k, v, state["cos"], state["sin"])
        else:
            out = attention(q, k, v, causal=case["causal"])
        return [out.detach(), *torch.autograd.grad(out, (q, k, v), state["dy"])]
    if kind == "flash":
        return flash_attention_forward(state["q"], state["k"], state["v"])
    if kind == "head":
        hidden, weight = state["hidden"], state["weight"]
        hidden.grad = weight.grad = None
        loss = ops.lm_head_cross_entropy(hidden, weight, state["targets"])
        loss.backward()
        return [loss.detach(), hidden.grad, weight.grad]
    if kind == "adamw":
        optimizer = state["optimizer"]
        optimizer.step()
        return [[p.detach(), optimizer.state[p]["m"], optimizer.state[p]["v"]] for p in state["params"]]
    raise ValueError(kind)


# ------------------------------------------------------------------------------ what a pass cannot do without
def _block_flops(case, tokens, seq):
    """(contractions outside attention, attention) of one block's forward pass over ``tokens`` tokens."""
    d, f = case["d_model"], case["d_ff"]
    dense = 2 * tokens * (d * (d + d // 2) + d * d + d * case["experts"]) + 2 * 6 * tokens * d * f
    return dense, 2 * tokens * seq * d


def _sizes(case):
    """(dense parameters outside embedding, expert parameters) of the decoder."""
    d, f = case["d_model"], case["d_ff"]
    dense = case["blocks"] * (d * (d + d // 2) + d * d + d * case["experts"] + 2 * d) + d * case["vocab"] + d
    return dense, case["blocks"] * case["experts"] * 3 * d * f


def work(case):
    kind = case["kind"]
    if kind in ("step", "logits"):
        tokens = case["batch"] * case["seq"]
        dense, attn = _block_flops(case, tokens, case["seq"])
        head = 2 * tokens * case["d_model"] * case["vocab"]
        n_dense, n_expert = _sizes(case)
        if kind == "logits":
            return {"bytes": 2 * (n_dense + n_expert) + 2 * tokens * (case["d_model"] + case["vocab"]),
                    "flops": case["blocks"] * (dense + attn) + head}
        state = 4 if case["expert_state"] == "float32" else 2
        table = case["vocab"] * case["d_model"]
        # the update reads and writes weights and both moments (dense: fp32 with a bf16 copy)
        return {"bytes": (n_dense + table) * (3 * 8 + 2) + n_expert * (2 * 2 + 4 * state),
                "flops": 3 * (case["blocks"] * dense + head) + 3.5 * case["blocks"] * attn}
    if kind == "moe":
        d, f, e, t = case["d_model"], case["d_ff"], case["experts"], case["tokens"]
        return {"bytes": 2 * e * 3 * d * f * 2 + 4 * 2 * t * d, "flops": 3 * (2 * 6 * t * d * f + 2 * t * d * e)}
    if kind == "ffn":
        d, f, t = case["d_model"], case["d_ff"], case["batch"] * case["seq"]
        return {"bytes": 2 * 9 * d * f * 2 + 4 * 2 * t * d, "flops": 3 * 3 * 6 * t * d * f}
    if kind in ("rope_attn", "attn"):
        B, S, H, Hkv = case["batch"], case["seq"], case["heads"], case["kv_heads"]
        causal = 0.5 if kind == "rope_attn" or case["causal"] else 1.0
        return {"bytes": 2 * B * S * HEAD_DIM * (4 * H + 4 * Hkv), "flops": 3.5 * 4 * B * H * S * S * HEAD_DIM * causal}
    if kind == "flash":
        B, S, H = case["batch"], case["seq"], case["heads"]
        return {"bytes": 2 * 4 * B * S * H * HEAD_DIM, "flops": 4 * B * H * S * S * HEAD_DIM}
    if kind == "head":
        t, d, v = case["tokens"], case["d_model"], case["vocab"]
        return {"bytes": 2 * (2 * t * d + 2 * v * d) + 8 * t, "flops": 3 * 2 * t * d * v}
    total = 0
    for shape, dtype in _adamw_shapes(case):
        width = 4 if dtype == torch.float32 else 2
        moment = 4 if dtype == torch.float32 or case["expert_state"] == "float32" else 2
        total += math.prod(shape) * (3 * width + 4 * moment)
    return {"bytes": total, "flops": 0}


# Measured on a B200: the native path against the plain PyTorch statements of the same operations on the GPU (other
# kernels, other summation order, intermediate roundings at other places), largest over the outputs and over the listed
# and some drawn cases; four times that is stated.
#   step       weights and loss after three steps at lr 1e-3: 0.005 to 0.03, at this rate a third of it.  AdamW's first
#              updates follow the sign of the gradient, so where a gradient is all rounding a weight moves the other way
#   logits     0.012, largest single difference 0.9: a token whose second and third expert are tied to within a bf16
#              rounding goes to another expert (0.03 is as much as a comparison can still use)
#   moe, ffn   0.005 with the same routing
#   attention  0.0033 (gradients), 0.0023 (fp16 inputs computed in bf16)
#   head       0.0004 (bf16 logits on both sides; up to 0.0013 where they stay in fp32)
#   adamw      0.0012 (bf16 moments; 1e-5 for fp32)
TOLERANCE = {
    "step": {"rel": 0.02, "max": 0.8}, "logits": {"rel": 0.03, "max": 0.95}, "moe": {"rel": 0.02}, "ffn": {"rel": 0.02},
    "rope_attn": {"rel": 0.013}, "attn": {"rel": 0.013}, "flash": {"rel": 0.01}, "head": {"rel": 0.005},
    "adamw": {"rel": 0.005},
}


def tolerance(case):
    return TOLERANCE[case["kind"]]


# ------------------------------------------------------------------------------ the same passes in 64 bits
def _swiglu64(x, w1, w2, w3):
    gate = x @ w1.t()
    return (gate * torch.sigmoid(gate) * (x @ w3.t())) @ w2.t()


def _attention64(state, causal, rotate):
    """Output and gradients of attention, one (sequence, KV head) at a time."""
    q, k, v, dy = (state[n].detach().double() for n in ("q", "k", "v", "dy"))
    B, S, H, Hkv = *q.shape[:3], k.shape[2]

    def turn(x, sign):
        """Rotates adjacent pairs of ``[S, ..., 128]`` by their position's angle."""
        if not rotate:
            return x
        cos, sin = (state[n][:S].double().view(S, *[1] * (x.dim() - 2), -1) for n in ("cos", "sin"))
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * cos - sign * b * sin, sign * a * sin + b * cos), -1).flatten(-2)

    out, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    hidden = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1) if causal else None
    for b in range(B):
        for j in range(Hkv):
            keys, values = turn(k[b, :, j], 1), v[b, :, j]
            dkeys, dvalues = torch.zeros_like(keys), torch.zeros_like(values)
            for h in range(j * (H // Hkv), (j + 1) * (H // Hkv)):
                queries, g = turn(q[b, :, h], 1), dy[b, :, h]
                p = queries @ keys.t() * HEAD_DIM ** -0.5
                if hidden is not None:
                    p.masked_fill_(hidden, -math.inf)
                p = p.softmax(-1)
                out[b, :, h] = p @ values
                dvalues += p.t() @ g
                ds = (g @ values.t() - (g * out[b, :, h]).sum(-1, keepdim=True)) * p * HEAD_DIM ** -0.5
                dq[b, :, h] = turn(ds @ keys, -1)
                dkeys += ds.t() @ queries
            dk[b, :, j], dv[b, :, j] = turn(dkeys, -1), dvalues
    return [out, dq, dk, dv]


def _moe64(x, router, w1, w2, w3):
    """Top-2 routed experts with renormalised weights; differentiable."""
    top, idx = (x @ router.t()).softmax(-1).topk(2, dim=-1)
    weights = top / top.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(w1.shape[0]):
        token, j = (idx == e).nonzero(as_tuple=True)
        out = out.index_add(0, token, _swiglu64(x[token], w1[e], w2[e], w3[e]) * weights[token, j, None])
    return out


def _norm64(x, weight):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * weight.double()


def _logits64(case, wrapped, ids):
    model, S, H = wrapped.module, case["seq"], case["heads"]

    def bf16(weight):      # the wrapped model computes with bf16 copies of its fp32 weights
        return weight.detach().to(BF16).double()

    angles = torch.arange(S, device="cuda").double()[:, None] * 10000.0 ** (
        -torch.arange(0, HEAD_DIM, 2, device="cuda").double() / HEAD_DIM)[None]
    x = bf16(model.token_embeddings.weight)[ids]
    B = x.shape[0]
    for layer in model.layers:
        n, a = _norm64(x, layer.ln1.weight), layer.attn
        heads = {name: (n @ bf16(getattr(a, name + "_proj").weight).t()).view(B, S, -1, HEAD_DIM) for name in "qkv"}
        state = {**heads, "dy": torch.zeros_like(heads["q"]), "cos": angles.cos(), "sin": angles.sin()}
        x = x + _attention64(state, True, True)[0].view(B, S, H * HEAD_DIM) @ bf16(a.output_proj.weight).t()
        n, f = _norm64(x, layer.ln2.weight).view(B * S, -1), layer.ffn
        experts = [p.detach().double() for p in (f.experts.w1, f.experts.w2, f.experts.w3)]
        x = x + _moe64(n, bf16(f.router.weight), *experts).view(x.shape)
    return _norm64(x, model.ln_final.weight) @ bf16(model.lm_head.weight).t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return None      # thousands of roundings in a row, then updates that follow the gradients' signs
    state = prepare(case, seed)
    if kind == "logits":
        with torch.no_grad():
            return _logits64(case, state["model"], state["x"])
    if kind == "moe":
        module = state["model"].module
        leaves = [state["x"], module.router.weight.to(BF16), module.experts.w1, module.experts.w2, module.experts.w3]
        leaves = [t.detach().double().requires_grad_(True) for t in leaves]
        out = _moe64(*leaves)
        dx, drouter, dw1, dw2, dw3 = torch.autograd.grad(out, leaves, state["dy"].double())
        return [out.detach(), dx, drouter, dw1, dw2, dw3]
    if kind == "ffn":
        params = list(state["model"].parameters())
        leaves = [t.detach().double().requires_grad_(True) for t in (state["x"], *params)]
        out = leaves[0]
        for w1, w2, w3 in zip(leaves[1::3], leaves[2::3], leaves[3::3]):
            out = _swiglu64(out, w1, w2, w3)
        return [out.detach(), *torch.autograd.grad(out, leaves, state["dy"].double())]
    if kind in ("rope_attn", "attn"):
        return _attention64(state, kind == "rope_attn" or case["causal"], kind == "rope_attn")
    if kind == "flash":
        q, k, v = (state[n].double() for n in "qkv")
        return torch.stack([(q[b] @ k[b].mT * HEAD_DIM ** -0.5).softmax(-1) @ v[b] for b in range(q.shape[0])])
    if kind == "head":
        hidden, weight = (state[n].detach().double().requires_grad_(True) for n in ("hidden", "weight"))
        loss = torch.nn.functional.cross_entropy(hidden @ weight.t(), state["targets"])
        return [loss.detach(), *torch.autograd.grad(loss, (hidden, weight))]
    results = []
    for p in state["params"]:      # first update of lr 1e-3, betas 0.9 and 0.999, eps 1e-8, decay 0.01
        g = p.grad.double()
        m, v = 0.1 * g, 0.001 * g * g
        step = 1e-3 * math.sqrt(1 - 0.999) / (1 - 0.9)
        results.append([p.detach().double() * (1 - 1e-3 * 0.01) - step * m / (v.sqrt() + 1e-8), m, v])
    return results
