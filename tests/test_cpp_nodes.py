"""The C++ autograd nodes against the Python nodes that they stand for."""
import os

import pytest
import torch

from b200moe.ops import native


def _nodes():
    module = native.nodes()
    if module is None:
        pytest.skip("built without PyTorch")
    return module


# ------------------------------------------------------------------------------ CPU
def test_nodes_leave_what_they_do_not_take_to_the_general_way():
    nodes = _nodes()
    x, w, word = torch.zeros(2, 128, 512, dtype=torch.bfloat16), torch.ones(512), torch.zeros(1, dtype=torch.int32)
    table, ids = torch.zeros(9, 512, dtype=torch.bfloat16), torch.zeros(3, dtype=torch.int64)
    grad, cos = torch.zeros(9, 512), torch.zeros(128, 64)
    assert nodes.rmsnorm(x, w, 1e-5, word) is None
    assert nodes.embedding(ids, table, grad) is None
    assert nodes.head(x, table, ids, grad, 1.0, 4096, word) is None
    square, fused = torch.zeros(512, 512), torch.zeros(768, 512)
    assert nodes.attn_half(x, w, fused.bfloat16(), fused, cos, cos, square.bfloat16(), square, w, word, 4, 1, 1e-5, 1e-5) is None
    experts = torch.zeros(2, 128, 512, dtype=torch.bfloat16)
    down = torch.zeros(2, 512, 128, dtype=torch.bfloat16)
    assert nodes.moe_layer(x, table[:2], experts, experts, down, None, grad[:2], experts.float(), experts.float(), down.float(), word,
                           256, False, False) is None
    with pytest.raises(RuntimeError, match="cannot load"):
        nodes.bind("/nonexistent/library.so")
    nodes.bind(native._LIB_PATH)


def test_transformations_that_look_through_nodes_get_the_python_ones():
    from torch.utils._python_dispatch import TorchDispatchMode

    from b200moe import ops

    class Other(torch.Tensor):
        pass

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    _nodes()
    x, seen = torch.zeros(2, 3), []
    assert ops.cpp_nodes(x, torch.nn.Parameter(x)) is native.nodes()
    assert ops.cpp_nodes(x, x.as_subclass(Other)) is None
    torch.func.vmap(lambda t: seen.append(ops.cpp_nodes(x)) or t)(x)
    torch.func.jvp(lambda t: seen.append(ops.cpp_nodes(x)) or t, (x,), (x,))
    with Watch():
        seen.append(ops.cpp_nodes(x))
    with torch.device("cpu"):
        seen.append(ops.cpp_nodes(x))
    native.set_nvtx(True)
    try:
        seen.append(ops.cpp_nodes(x))
    finally:
        native.set_nvtx(False)
    assert seen == [None] * 5


def test_library_is_built_where_the_nodes_do_not_compile(monkeypatch, tmp_path, capsys):
    import subprocess

    from b200moe import build
    run, out = subprocess.run, tmp_path / "_C"
    out.mkdir()
    stale = out / "b200moe_nodes.so"
    for path in (stale, out / "b200moe_nodes.so.sha"):
        path.write_text("of another build")

    def without_compiler(cmd, **kwargs):
        return run(["false"], **kwargs) if cmd[0] == "g++" else run(cmd, **kwargs)

    monkeypatch.setattr(build, "HERE", str(tmp_path))
    monkeypatch.setattr(build, "OUT", str(out))
    monkeypatch.setattr(build, "LIB", str(out / "lib.so"))
    monkeypatch.setattr(build, "_sources", lambda: ["pp_link.cu"])
    monkeypatch.setattr(build.subprocess, "run", without_compiler)
    build.build_all()
    assert os.path.getsize(build.LIB) > 0 and not stale.exists() and not (out / "b200moe_nodes.so.sha").exists()
    assert "C++ autograd nodes not built" in capsys.readouterr().err


def test_nodes_that_do_not_load_leave_the_python_ones(monkeypatch, tmp_path):
    (tmp_path / "_C").mkdir()
    (tmp_path / "_C" / "b200moe_nodes.so").write_bytes(b"no library")
    native.require()
    monkeypatch.setattr(native, "_HERE", str(tmp_path))
    monkeypatch.setattr(native, "_nodes", None)
    with pytest.warns(UserWarning, match="does not load"):
        assert native.nodes() is None
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("error")       # said once
        assert native.nodes() is None


def test_refused_launch_is_named_as_the_python_bindings_name_it():
    import ctypes
    nodes, lib = _nodes(), native.require()
    nodes.check(0, None, 0)
    with pytest.raises(RuntimeError, match=r"^b2_attention_fwd_ex failed with code -12 \(tensor map k: driver result 0\)"):
        nodes.check(-12, "b2_attention_fwd_ex", 1)
    # rows of 65 * 128 columns: the first launch of the sequence is refused before anything touches a device
    null, pointers = ctypes.c_void_p(0), 14
    code = lib.b2_attn_half_fwd(*[null] * pointers, *[ctypes.c_int(v) for v in (1, 128, 65, 65)], ctypes.c_float(1e-5),
                                ctypes.c_float(1e-5), null, null)
    with pytest.raises(RuntimeError, match="^b2_rmsnorm_fwd failed with code -10"):
        nodes.check(code, None, 1)


# ------------------------------------------------------------------------------ GPU
def _rel(a, b):
    return float((a.double() - b.double()).norm() / (b.double().norm() + 1e-30))


def _decoder(D=512, heads=4, experts=4, ffn=256, vocab=320, blocks=2, expert_grad=torch.float32):
    from b200moe.models import TransformerLMPipelined
    from b200moe.parallel import FSDPWrapperPipelined
    torch.manual_seed(3)
    with torch.device("cuda"):
        model = TransformerLMPipelined(vocab, 256, D, blocks, heads, 0, 1, num_expert_per_node=experts, d_ff=ffn)
    return FSDPWrapperPipelined(model, None, None, compute_dtype=torch.bfloat16, expert_grad_dtype=expert_grad)


def _step(model, ids, aux=0.0, scale=0.5):
    model.clear_grad_accumulators()
    out = model.loss(ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), return_aux_loss=aux > 0, grad_scale=scale)
    loss, extra = out if aux else (out, None)
    torch.autograd.backward([loss] + ([extra] if aux else []), [torch.full_like(loss, scale)] + ([torch.full_like(loss, aux)] if aux else []))
    model.reduce_accumulated_gradients()
    grads = {n: (p.main_grad if hasattr(p, "main_grad") else p.grad).clone() for n, p in model.named_parameters()}
    return loss.detach().clone(), extra, grads


@pytest.mark.gpu
@pytest.mark.parametrize("S,aux,expert_grad,recompute", [(128, 0.0, torch.float32, False), (256, 0.02, torch.bfloat16, False),
                                                         (128, 0.02, torch.float32, True)])
def test_training_step_on_cpp_nodes_matches_python_nodes(monkeypatch, S, aux, expert_grad, recompute):
    _nodes()
    model = _decoder(expert_grad=expert_grad)
    for layer in model.module.layers:
        layer.ffn.recompute = recompute
    ids = torch.randint(0, 320, (3, S + 1), device="cuda")
    before = native.launch_count()
    loss, extra, got = _step(model, ids, aux)
    launched = native.launch_count() - before
    monkeypatch.setattr(native, "nodes", lambda: None)
    before = native.launch_count()
    want_loss, want_extra, want = _step(model, ids, aux)
    assert launched == native.launch_count() - before > 50
    # the same forward kernels; the loss is summed in a double, whose additions' order does not reach the fp32 result
    assert torch.equal(loss, want_loss)
    assert extra is None or torch.equal(extra, want_extra)
    # backward: the sum of a block's two input gradients is rounded once where it was rounded twice (2^-9 each); node by node below
    assert got.keys() == want.keys() and all(_rel(got[n], want[n]) < 2e-2 for n in want)
    with torch.no_grad():
        logits = model(ids[:, :-1].contiguous())
        monkeypatch.undo()
        assert torch.equal(model(ids[:, :-1].contiguous()), logits)
    native.check_status()


def _weight(*shape, scale, grad=torch.float32):
    w = (torch.randn(*shape, device="cuda") * scale).bfloat16().requires_grad_(True)
    w.main_grad = torch.zeros(*shape, dtype=grad, device="cuda")
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("E,residual,recompute,used,grad", [
    (4, True, False, "both", torch.float32), (4, False, False, "out", torch.float32), (4, True, True, "out", torch.bfloat16),
    (4, True, False, "aux", torch.float32), (4, False, True, "aux", torch.bfloat16), (12, True, False, "both", torch.bfloat16),
    (16, False, False, "both", torch.float32), (2, True, False, "both", torch.float32)])
@pytest.mark.parametrize("T", [1, 300])
def test_routed_layer_node_gives_the_bits_of_the_python_node(T, E, residual, recompute, used, grad):
    from b200moe.ops import moe_fused
    _nodes()
    torch.manual_seed(E)
    D, F = 256, 384
    router = _weight(E, D, scale=D ** -0.5)
    w1, w3, w2 = _weight(E, F, D, scale=D ** -0.5, grad=grad), _weight(E, F, D, scale=D ** -0.5, grad=grad), _weight(E, D, F, scale=F ** -0.5, grad=grad)
    x = torch.randn(T, D, device="cuda").bfloat16().requires_grad_(True)
    res = torch.randn(T, D, device="cuda").bfloat16().requires_grad_(True) if residual else None
    dout, daux = torch.randn(T, D, device="cuda").bfloat16(), torch.tensor(0.3, device="cuda")
    results = []
    for call in (moe_fused.moe_layer_node, moe_fused.moe_layer_fused):
        for w in (router, w1, w3, w2):
            w.main_grad.zero_()
        out, aux = call(x, router, w1, w2, w3, res, recompute=recompute, balance=True)
        outputs, douts = [], []
        if used != "aux":
            outputs, douts = [out], [dout]
        if used != "out":
            outputs, douts = outputs + [aux], douts + [daux]
        inputs = [x] + ([res] if residual and used != "aux" else [])
        for again in (True, False):                # a retained graph gives the same once more
            grads = torch.autograd.grad(outputs, inputs, douts, retain_graph=again)
        results.append(([out, aux, *grads, w1.main_grad.clone(), w3.main_grad.clone(), w2.main_grad.clone()], router.main_grad.clone()))
    (cpp, crouter), (python, prouter) = results
    assert all(torch.equal(a, b) for a, b in zip(cpp, python))
    assert _rel(crouter, prouter) < 1e-5           # fp32 sums in the order of atomic additions
    assert bool(crouter.any()) and bool(cpp[2].any()) and (used == "aux" or bool(cpp[-1].any()))
    native.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,used", [(2, 256, "both"), (3, 128, "sum"), (3, 128, "normed"), (1, 4096, "both")])
def test_attention_half_node_against_64_bits(B, S, used):
    """Both outputs and all gradients, no further from 64 bits than the separate nodes; one output unused; twice through a retained
    graph."""
    from b200moe import ops
    from b200moe.ops import functional as Fn
    from b200moe.ops.attention import fused_qkv_attention
    from b200moe.ops.block import attn_half
    _nodes()
    torch.manual_seed(S)
    hq, hkv, D = 4, 1, 512
    x = torch.randn(B, S, D, device="cuda").bfloat16().requires_grad_(True)
    ln1, ln2 = ((torch.rand(D, device="cuda") + 0.5).requires_grad_(True) for _ in range(2))
    wqkv, wo = _weight((hq + 2 * hkv) * 128, D, scale=1.5 * D ** -0.5), _weight(D, D, scale=D ** -0.5)
    cos, sin = Fn.rope_tables(10000.0, 128, S, "cuda")
    dsum, dnormed = torch.randn(B, S, D, device="cuda").bfloat16(), torch.randn(B, S, D, device="cuda").bfloat16()

    def separate():
        qkv = ops.linear_rope(ops.rmsnorm(x, ln1, 1e-5).view(B * S, D), wqkv, cos, sin, (hq + hkv) * 128, S)
        out = ops.linear(fused_qkv_attention(qkv, B, S, hq, hkv, 128, cos, sin, pre_rotated=True).reshape(B, S, D), wo)
        return ops.add_rmsnorm(x, out, ln2, 1e-5)

    def whole():
        return attn_half(x, ln1, wqkv, cos, sin, wo, ln2, (hq, hkv), 1e-5, 1e-5)

    def exact():
        leaves = [t.detach().double().requires_grad_(True) for t in (x, ln1, wqkv, wo, ln2)]
        x64, g1, wq64, wo64, g2 = leaves
        norm = lambda t, g: t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-5) * g  # noqa: E731
        q, k, v = (t.view(B, S, -1, 128) for t in (norm(x64, g1) @ wq64.t()).split((hq * 128, hkv * 128, hkv * 128), -1))
        c, s = (t.double().view(S, 1, 64) for t in (cos, sin))

        def turn(t):
            a, b = t[..., 0::2], t[..., 1::2]
            return torch.stack((a * c - b * s, a * s + b * c), -1).flatten(-2)

        q, k, v = (t.transpose(1, 2) for t in (turn(q), turn(k), v))
        scores = q @ k.mT * 128 ** -0.5
        scores = scores.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), -float("inf"))
        total = x64 + (scores.softmax(-1) @ v).transpose(1, 2).reshape(B, S, D) @ wo64.t()
        return (total, norm(total, g2)), leaves

    def select(pair):
        return {"both": pair, "sum": pair[:1], "normed": pair[1:]}[used]

    douts = select((dsum, dnormed))
    (total, normed), leaves = exact()
    # gradients that the outputs in use do not reach count as zeros
    want = [total, normed, *torch.autograd.grad(select((total, normed)), leaves, [d.double() for d in douts], allow_unused=True, materialize_grads=True)]
    found = []
    for call in (whole, separate):
        for repeat in (False, True):
            wqkv.main_grad.zero_(), wo.main_grad.zero_()
            pair = call()
            for again in ((True, False) if repeat else (False,)):
                dx, d1, d2 = torch.autograd.grad(select(pair), (x, ln1, ln2), douts, retain_graph=again, allow_unused=True, materialize_grads=True)
            got = [*pair, dx, d1, wqkv.main_grad / (1 + repeat), wo.main_grad / (1 + repeat), d2]
            if repeat:
                assert all(torch.equal(a, b) for a, b in zip(got, found[-1]))
            else:
                found.append([t.detach().clone() for t in got])
    assert torch.equal(found[0][0], found[1][0]) and torch.equal(found[0][1], found[1][1])      # the same forward kernels
    for cpp, python, w in zip(found[0], found[1], want):
        # four roundings to bf16 (2^-9 at most, a third of it in the mean) lie between input and output of this half each way, the
        # probabilities' and dS' among them
        assert _rel(cpp, w) < 1e-2 and _rel(cpp, w) <= 1.05 * _rel(python, w) + 1e-5
    native.check_status()


@pytest.mark.gpu
def test_cpp_nodes_under_saved_tensor_hooks_and_on_another_stream():
    _nodes()
    model = _decoder()
    ids = torch.randint(0, 320, (2, 129), device="cuda")
    _, _, want = _step(model, ids)
    with torch.autograd.graph.save_on_cpu():
        _, _, got = _step(model, ids)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _, _, other = _step(model, ids)
    torch.cuda.current_stream().wait_stream(side)
    # sums of atomics (router, embedding) differ in their last bits
    assert all(_rel(got[n], want[n]) < 1e-3 and _rel(other[n], want[n]) < 1e-3 for n in want)
    native.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["ln1", "attn", "attn.output_proj", "ffn", "ffn.router"])
def test_watched_modules_are_called(which):
    model = _decoder(blocks=1)
    ids = torch.randint(0, 320, (2, 128), device="cuda")
    calls = []
    layer = model.module.layers[0]
    handle = layer.get_submodule(which).register_forward_hook(lambda *_: calls.append(1))
    with torch.no_grad():
        model(ids)
        handle.remove()
        model(ids)
    assert calls == [1]


@pytest.mark.gpu
@pytest.mark.parametrize("T,D,V,chunk", [(1, 64, 64, 4096), (300, 512, 320, 128), (257, 128, 32000, 256)])
def test_head_node_in_chunks(monkeypatch, T, D, V, chunk):
    from b200moe import ops
    from b200moe.ops import loss as L
    _nodes()
    monkeypatch.setattr(L, "CHUNK_TOKENS", chunk)
    hidden = torch.randn(T, D, device="cuda").bfloat16().requires_grad_(True)
    weight = (torch.randn(V, D, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    weight.main_grad = torch.zeros(V, D, device="cuda")
    targets = torch.randint(0, V, (T,), device="cuda")
    out = []
    for _ in range(2):
        hidden.grad = None
        weight.main_grad.zero_()
        loss = ops.lm_head_cross_entropy(hidden, weight, targets, 0.25)
        (loss * 0.5).backward()                       # another factor than announced: dh follows, dW keeps its word
        out.append((loss.detach(), hidden.grad, weight.main_grad.clone()))
        monkeypatch.setattr(native, "nodes", lambda: None)
    for a, b in zip(*out):
        assert _rel(a, b) < 1e-5
    assert weight.grad is None
    native.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("cpp", [True, False])
def test_head_with_a_known_factor_twice_through_one_graph(monkeypatch, cpp):
    from b200moe import ops
    _nodes()
    if not cpp:
        monkeypatch.setattr(native, "nodes", lambda: None)
    hidden = torch.randn(70, 128, device="cuda").bfloat16().requires_grad_(True)
    weight = (torch.randn(320, 128, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    weight.main_grad = torch.zeros(320, 128, device="cuda")
    targets = torch.randint(0, 320, (70,), device="cuda")
    loss = ops.lm_head_cross_entropy(hidden, weight, targets, 0.25)
    summed = weight.main_grad.clone()
    grads = [torch.autograd.grad(loss, hidden, torch.full_like(loss, f), retain_graph=f < 1)[0].clone() for f in (0.5, 0.25, 0.5, 1.0)]
    # powers of two: exact; the announced factor is already in dh, and the weight's gradient is added by the forward pass alone
    assert torch.equal(grads[0], 2 * grads[1]) and torch.equal(grads[0], grads[2]) and torch.equal(grads[3], 4 * grads[1])
    assert bool(grads[1].any()) and torch.equal(weight.main_grad, summed)
    native.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradient_buffers_are_those_of_the_backward_pass(dtype):
    """A ``main_grad`` replaced between the passes is followed; one that is taken away leaves an ordinary gradient."""
    _nodes()
    model = _decoder(blocks=1)
    inner = model.module.layers[0]
    weights = [model.module.token_embeddings.compute_weight, inner.attn.qkv_weight, inner.attn.output_proj.compute_weight,
               inner.ffn.router.compute_weight, inner.ffn.experts.w1, inner.ffn.experts.w3, inner.ffn.experts.w2]
    ids = torch.randint(0, 320, (2, 129), device="cuda")

    def run(change):
        model.clear_grad_accumulators()
        old = [w.main_grad for w in weights]
        loss = model.loss(ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), grad_scale=1.0)
        change()
        loss.backward()
        got = [w.main_grad if hasattr(w, "main_grad") else w.grad for w in weights]
        untouched = not any(bool(o.any()) for o in old)
        for w, o in zip(weights, old):
            w.main_grad, w.grad = o, None
        return [g.clone() for g in got], untouched

    def swap():
        for w in weights:
            w.main_grad = torch.zeros_like(w.main_grad, dtype=dtype)

    def remove():
        for w in weights[1:]:                      # (the table of the embedding does not ask for a gradient of its own)
            del w.main_grad

    kept, _ = run(lambda: None)
    for change in (swap, remove):
        got, untouched = run(change)
        assert untouched or change is remove
        assert len(got) == 7 and all(_rel(g, k) < (5e-3 if g.dtype == torch.bfloat16 else 1e-4) for g, k in zip(got, kept))
    native.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("part,recompute", [("attention", False), ("experts", False), ("experts", True)])
def test_backward_passes_hold_no_more_memory_than_the_python_nodes(monkeypatch, part, recompute):
    from b200moe import ops
    _nodes()
    layer = _decoder(D=1024, heads=8, ffn=3584, blocks=1, expert_grad=torch.bfloat16).module.layers[0]
    layer.ffn.recompute = recompute
    x = torch.randn(16, 256, 1024, device="cuda").bfloat16().requires_grad_(True)

    def outputs():
        if part == "experts":
            return (layer.ffn(x),)
        half = layer._attention_half(x)
        return half if half is not None else ops.add_rmsnorm(x, layer.attn(layer.ln1(x)), layer.ln2.weight, layer.ln2.eps)

    peaks, grads = [], []
    for _ in range(2):
        out = outputs()
        douts = [torch.full_like(o, 0.01) for o in out]
        torch.cuda.synchronize()
        torch.cuda.empty_cache()                        # (blocks left by others may be larger than what is asked for)
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        grads.append(torch.autograd.grad(out, x, douts)[0])
        torch.cuda.synchronize()
        peaks.append(torch.cuda.max_memory_allocated() - before)
        del out, douts
        monkeypatch.setattr(native, "nodes", lambda: None)
    assert peaks[0] <= peaks[1] + (2 << 20), peaks      # the allocator's granularity
    assert _rel(*grads) < 1e-2
    native.check_status()
