"""ctypes bindings of the in-tree sm_100a library ``b200moe/_C/libb200moe.so``.

Every function takes torch tensors, launches on the current CUDA stream and
returns torch tensors.  ``has(op)`` tells the op layer whether the kernel family
``op`` is loaded; ``require()`` raises if the library is missing, so a GPU run
can never fall back silently.  ``launch_count()`` counts launches of this
library's kernels (the benchmark reports it).
"""
from __future__ import annotations

import ctypes
import os

import torch

_HERE = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# B200MOE_DEBUG=1 loads the checked build (``B200MOE_DEBUG=1 python -m b200moe.build``): data-dependent indices
# are range-checked in the kernels and ``check_status`` also raises on a recorded violation.
_DEBUG = os.environ.get("B200MOE_DEBUG", "0") not in ("", "0")
_LIB_PATH = (os.path.join(_HERE, "_C", "debug", "libb200moe_debug.so") if _DEBUG
             else os.path.join(_HERE, "_C", "libb200moe.so"))
_lib = None
_load_error = None
_launches = 0
_status = {}
_entries = {}        # entry point name -> ctypes function
_has = {}            # op family -> whether the library has it

_FAMILIES = {
    "gemm": "b2_gemm_nt", "rmsnorm": "b2_rmsnorm_fwd", "router": "b2_router_top2_fwd",
    "lmhead_ce": "b2_cross_entropy2", "adamw": "b2_adamw", "embedding": "b2_embedding_fwd",
    "rope": "b2_rope", "moe": "b2_moe_plan", "attention": "b2_attention_fwd_ex", "comm": "b2_comm_allreduce",
    "swiglu": "b2_swiglu_bwd", "zero": "b2_zero",
}


def _load():
    global _lib, _load_error
    if _lib is not None or _load_error is not None:
        return _lib
    if not os.path.exists(_LIB_PATH):
        _load_error = f"{_LIB_PATH} not found; run `python -m b200moe.build`"
        return None
    try:
        _lib = ctypes.CDLL(_LIB_PATH)
    except OSError as error:
        _load_error = str(error)
        _lib = None
        return None
    mode = os.environ.get("B200MOE_GEMM_TILE_MODE")
    if mode:          # A/B runs of whole programs: see set_gemm_tile_mode
        _lib.b2_gemm_set_tile_mode(ctypes.c_int(int(mode)))
    return _lib


def require():
    if _load() is None:
        raise RuntimeError(f"b200moe native library unavailable: {_load_error}")
    return _lib


def has(op: str) -> bool:
    known = _has.get(op)
    if known is None:
        lib = _load()
        symbol = _FAMILIES.get(op)
        known = lib is not None and symbol is not None and hasattr(lib, symbol)
        if lib is not None:
            _has[op] = known
    return known


def available_ops() -> list:
    return sorted(op for op in _FAMILIES if has(op))


def launch_count() -> int:
    return _launches + (_nodes.launches() if _nodes else 0)


def count_launch(n: int = 1) -> None:
    """For callers that launch through ``require()`` directly."""
    global _launches
    _launches += n


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


# Stream and device as plain integers: ``torch.cuda.current_stream()`` builds two objects and looks the device up three
# times, which was a quarter of the host time of a small training step.
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_raw_device = getattr(torch._C, "_cuda_getDevice", None)


def _stream():
    return ctypes.c_void_p(_raw_stream(_raw_device()))


_nodes = None        # the C++ autograd nodes (csrc/nodes.cpp), False where there are none


def _load_nodes():
    """The extension, bound to this library; ``False``, with a warning, where it was not built or does not fit the
    installed PyTorch."""
    import importlib.machinery
    import importlib.util
    import warnings
    path = os.path.join(_HERE, "_C", "b200moe_nodes.so")
    reason = "not found"
    if os.path.exists(path):
        loader = importlib.machinery.ExtensionFileLoader("b200moe_nodes", path)
        try:
            module = importlib.util.module_from_spec(importlib.util.spec_from_loader("b200moe_nodes", loader))
            loader.exec_module(module)
            module.bind(_LIB_PATH)
            return module
        except (ImportError, RuntimeError) as error:
            reason = f"does not load ({error})"
    warnings.warn(f"{path} {reason}: small layers run at the speed of Python; run `python -m b200moe.build`")
    return False


def nodes():
    """The C++ autograd nodes; ``None`` where there are none (the nodes in Python then issue the same launches) and while
    launches are timed or marked one by one."""
    global _nodes
    if _nodes is None:
        require()
        _nodes = _load_nodes()
    return _nodes if _nodes and _timed is None and not _nvtx else None


def status_word(device=None) -> torch.Tensor:
    """Device int32 word that kernels set non-zero when a bounded wait ran out."""
    word = _status.get(device) if type(device) is torch.device else None
    if word is not None:
        return word
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    word = _status.get(device)
    if word is None:
        word = torch.zeros(1, dtype=torch.int32, device=device)
        _status[device] = word
    return word


def debug_records(clear: bool = False) -> dict:
    """Checked build only: the first range violation recorded by each source file, as
    ``{file: (code, value, bound, block)}``; empty in the normal build."""
    lib = _load()
    found = {}
    if lib is None:
        return found
    for name in ("moe", "comm", "moe_ep"):
        reader = getattr(lib, f"b2_{name}_debug_read", None) if _DEBUG else None
        if reader is None:
            continue
        record = (ctypes.c_int * 4)()
        if reader(record, ctypes.c_int(int(clear))) == 0 and record[0]:
            found[name] = tuple(record)
    return found


def set_wait_seconds(seconds: float) -> None:
    """Budget of every cross-GPU wait inside this library's kernels on the current device (default 10 s).  A wait
    that runs out makes its kernel skip the dependent work, set the status word and return."""
    rc = require().b2_comm_set_wait_ns(ctypes.c_longlong(int(float(seconds) * 1e9)))
    if rc != 0:
        raise RuntimeError(f"b2_comm_set_wait_ns failed with code {rc}")


def clear_status(device=None) -> None:
    """Reset the status word after a reported failure has been handled (tests; a trainer restarts instead)."""
    status_word(device).zero_()


def check_status() -> int:
    """Synchronising read of the status word; raises if a kernel gave up (or, in the checked build, if a kernel
    recorded an out-of-range index)."""
    value = int(status_word().item())
    if value:
        raise RuntimeError(f"b200moe kernel reported wait timeout code {value}")
    if _DEBUG:
        bad = debug_records()
        if bad:
            raise RuntimeError(f"b200moe checked build recorded out-of-range indices: {bad}")
    return value


_nvtx = False


def set_nvtx(enabled: bool) -> None:
    """Wrap every launch of this library in an NVTX range named after its entry point (for Nsight Systems
    timelines; the trainer switches it on with ``profile.enabled``)."""
    global _nvtx
    _nvtx = bool(enabled)


_timed = None      # list of (label, start event, end event) while launch timing is on


def start_launch_timing() -> None:
    """Bracket every launch of this library with a pair of CUDA events on its stream (``launch_times`` reads them).
    For per-kernel time tables of a whole step; it adds two event records per launch, so timed regions of a
    benchmark leave it off."""
    global _timed
    _timed = []


def launch_times() -> dict:
    """Stops launch timing and returns ``{label: (launches, total ms)}``; synchronises the device."""
    global _timed
    records, _timed = _timed or [], None
    torch.cuda.synchronize()
    table: dict = {}
    for label, begin, end in records:
        count, total = table.get(label, (0, 0.0))
        table[label] = (count + 1, total + begin.elapsed_time(end))
    return table


def _call(name, *args, n: int = 1, tag: str = ""):
    global _launches
    entry = _entries.get(name)
    if entry is None:
        entry = _entries[name] = getattr(require(), name)
    if _timed is None and not _nvtx:
        rc = entry(*args)
        if rc != 0:
            raise RuntimeError(f"{name} failed with code {rc}{_failure_detail(name, rc)}")
        _launches += n
        return
    if _timed is not None:
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        rc = entry(*args)
        end.record()
        _timed.append((f"{name} {tag}".strip(), begin, end))
        if rc != 0:
            raise RuntimeError(f"{name} failed with code {rc}")
        _launches += n
        return
    torch.cuda.nvtx.range_push(name)
    try:
        rc = entry(*args)
    finally:
        torch.cuda.nvtx.range_pop()
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc}{_failure_detail(name, rc)}")
    _launches += n


def _failure_detail(name: str, rc: int) -> str:
    """What else is known about a refused launch (the attention entry points keep the driver's result of a
    tensor-map encode that failed)."""
    if name.startswith("b2_attention") and -14 <= rc <= -11:
        reader = getattr(_lib, "b2_attention_last_encode_result", None)
        if reader is not None:
            return f" (tensor map {('q', 'k', 'v', 'dout')[-11 - rc]}: driver result {reader()})"
    return ""


_I, _L, _F = ctypes.c_int, ctypes.c_longlong, ctypes.c_float


def _bf16(t):
    if t.dtype != torch.bfloat16:
        raise TypeError(f"expected bfloat16, got {t.dtype}")
    return t


# ------------------------------------------------------------------------------ GEMM
def set_gemm_tile_mode(mode: int) -> None:
    """0: automatic (the default): 128x64 or 128x128 tiles for products of one or two waves, 256x256 tiles on one CTA for
    reductions of 6144 and more over at least two such tiles per SM, else on CTA pairs (``cta_group::2``) where they fill
    the machine, else 128x256 tiles; 1: always 128x256 CTA tiles; 2: single-CTA 256x256 tiles wherever legal; 3: CTA pairs
    wherever legal; 4: like 0, the expert-parallel return included; 5: automatic among the single-CTA kinds; 6, 7: 128x128
    and 128x64 tiles.  The environment variable ``B200MOE_GEMM_TILE_MODE`` sets it at
    load time."""
    require().b2_gemm_set_tile_mode(_I(mode))


def gemm_nt(x, w, out_dtype=None, tile_expert=None, num_m_tiles=None, num_experts: int = 1, align256: bool = False):
    """``x [M,K] @ w[e] [N,K]ᵀ``.  Rows of ``w`` below 17: skinny path, fp32 result."""
    M, K = x.shape
    N = w.shape[-2]
    if N <= 16 and num_experts == 1:
        out = torch.empty(M, N, dtype=torch.float32, device=x.device)
        _call("b2_skinny_nt", _p(_bf16(x)), _p(_bf16(w)), _p(out), _I(M), _I(N), _I(K), _stream())
        return out
    out_dtype = out_dtype or torch.bfloat16
    out = torch.empty(M, N, dtype=out_dtype, device=x.device)
    assert x.stride(-1) == 1 and w.is_contiguous()
    _call("b2_gemm_nt", _p(_bf16(x)), _p(_bf16(w)), _p(out), _I(M), _I(N), _I(K), _L(x.stride(0)), _L(K), _L(N),
          _I(num_experts), _p(tile_expert), _p(num_m_tiles), _I(int(align256)),
          _I(0 if out_dtype == torch.bfloat16 else 4),
          _p(status_word(x.device)), _stream(), tag=f"{'grouped ' if tile_expert is not None else ''}N={N} K={K}")
    return out


def gemm_nt_rope(x, w, cos, sin, rope_cols: int, seq: int):
    """``x [M,K] @ w [N,K]ᵀ`` with the rotary embedding applied, in the GEMM epilogue, to output columns
    ``[0, rope_cols)``: heads of 128 columns, adjacent pairs, position ``row mod seq``; ``cos``/``sin`` fp32
    ``[>=seq, 64]``."""
    M, K = x.shape
    N = w.shape[0]
    if cos.shape[-1] != 64 or cos.dtype != torch.float32 or not cos.is_contiguous() or cos.shape[0] < seq:
        raise ValueError("rotary tables must be contiguous fp32 [>= seq, 64] (head_dim 128)")
    out = torch.empty(M, N, dtype=torch.bfloat16, device=x.device)
    assert x.stride(-1) == 1 and w.is_contiguous()
    _call("b2_gemm_nt_rope", _p(_bf16(x)), _p(_bf16(w)), _p(out), _I(M), _I(N), _I(K), _L(x.stride(0)), _L(N),
          _p(cos), _p(sin), _I(rope_cols), _I(seq), _p(status_word(x.device)), _stream())
    return out


def gemm_nn(dy, w, w2=None, tile_expert=None, num_m_tiles=None, num_experts: int = 1, align256: bool = False,
            out=None, alpha=None):
    """``dy [M,K] @ w[e] [K,N]`` (``w`` rows are the reduction index).  With ``w2``
    the reduction continues over ``w2``'s rows: ``dy = [a | b]``, result ``a w + b w2``.  ``alpha``: fp32 device scalar
    that multiplies the result in the epilogue."""
    M, K = dy.shape
    N = w.shape[-1]
    if K <= 16 and num_experts == 1 and w2 is None and alpha is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=dy.device)
        _call("b2_skinny_nn", _p(dy.float().contiguous()), _p(_bf16(w)), _p(out), _I(M), _I(K), _I(N), _stream())
        return out
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=dy.device)
    k_split = w.shape[-2] if w2 is not None else 0
    assert dy.stride(-1) == 1 and w.is_contiguous() and out.stride(-1) == 1 and out.shape == (M, N)
    _call("b2_gemm_nn", _p(_bf16(dy)), _p(_bf16(w)), _p(w2), _p(_bf16(out)), _I(M), _I(N), _I(K), _I(k_split),
          _L(dy.stride(0)), _L(N), _L(out.stride(0)), _I(num_experts), _p(tile_expert), _p(num_m_tiles), _I(int(align256)),
          _p(alpha), _p(status_word(dy.device)), _stream(),
          tag=f"{'grouped ' if tile_expert is not None else ''}N={N} K={K}")
    return out


def swiglu_bwd_in_product(M: int, F: int, K: int) -> bool:
    """Whether ``gemm_nn_swiglu_bwd`` is one launch."""
    return bool(require().b2_swiglu_bwd_in_product(_L(M), _I(F), _I(K)))


def gemm_nn_swiglu_bwd(dy, w, gate, up, tile_expert=None, num_m_tiles=None, num_experts: int = 1,
                       align256: bool = False, live_rows=None):
    """``dh = dy [M,K] @ w[e] [K,F]`` and the SwiGLU backward of it: returns ``dgu [M,2F]`` (gradients of the gate and up
    pre-activations) and ``h = silu(gate) * up [M,F]``.

    One launch, ``dh`` never stored, where the reduction is long enough to hide the five tensors of the epilogue
    (4096 x 14336, K 4096: 436 us against 478 us; 6001 x 32000, K 2048: 1067 against 1208) or where launches count
    (1024 x 1536, K 512: 22 against 31).  In between the product and an elementwise kernel are faster (8192 x 3584, K
    1024: 114 us against 130 us; 4096 x 1536, K 1024: 34 against 40)."""
    M, K = dy.shape
    F = w.shape[-1]
    if not swiglu_bwd_in_product(M, F, K):
        dh = gemm_nn(dy, w, tile_expert=tile_expert, num_m_tiles=num_m_tiles, num_experts=num_experts,
                     align256=align256)
        return swiglu_bwd(dh, gate, up, live_rows=live_rows)
    dgu = torch.empty(M, 2 * F, dtype=torch.bfloat16, device=dy.device)
    h = torch.empty(M, F, dtype=torch.bfloat16, device=dy.device)
    assert dy.stride(-1) == 1 and w.is_contiguous() and gate.is_contiguous() and up.is_contiguous()
    assert gate.shape == up.shape == (M, F)
    _call("b2_gemm_nn_swiglu_bwd", _p(_bf16(dy)), _p(_bf16(w)), _p(_bf16(gate)), _p(_bf16(up)), _p(dgu), _p(h), _I(M),
          _I(F), _I(K), _L(dy.stride(0)), _I(num_experts), _p(tile_expert), _p(num_m_tiles), _I(int(align256)),
          _p(status_word(dy.device)), _stream())
    return dgu, h


def gemm_tn(dy, x, out=None, accumulate: bool = False, out_dtype=None, expert_offsets=None, num_experts: int = 1,
            alpha=None, counts=None):
    """``out[e] (+)= dy[rows_e]ᵀ @ x[rows_e]`` -> ``[E?, N_out, K_in]``; fp32 or bf16 output.  ``alpha``: fp32 device
    scalar that multiplies the product.  ``counts``: int32 ``[E]`` rows of each segment that are not zero padding."""
    R, M = dy.shape
    N = x.shape[1]
    if M <= 16 and expert_offsets is None and alpha is None:
        if out is None:
            out = torch.zeros(M, N, dtype=torch.float32, device=dy.device)
            accumulate = True
        if out.dtype != torch.float32:
            raise TypeError("skinny weight gradients accumulate in fp32")
        if not accumulate:
            out.zero_()
        _call("b2_skinny_tn", _p(dy.float().contiguous()), _p(_bf16(x)), _p(out), _I(R), _I(M), _I(N), _stream())
        return out if out_dtype is None else out.to(out_dtype)
    want = None
    if out is None:
        want = out_dtype or torch.float32
        store = torch.float32 if want not in (torch.float32, torch.bfloat16) else want
        shape = (num_experts, M, N) if expert_offsets is not None else (M, N)
        out = torch.empty(shape, dtype=store, device=dy.device)
        accumulate = False
    kind = 1 if out.dtype == torch.float32 else 2
    assert dy.stride(-1) == 1 and x.stride(-1) == 1 and out.is_contiguous()
    _call("b2_gemm_tn", _p(_bf16(dy)), _p(_bf16(x)), _p(out), _p(None), _I(0), _I(M), _I(N), _I(R), _L(dy.stride(0)),
          _L(x.stride(0)), _L(N), _I(num_experts), _p(expert_offsets), _p(counts), _I(kind), _F(1.0 if accumulate else 0.0),
          _p(alpha), _p(status_word(dy.device)), _stream(),
          tag=f"{'grouped ' if expert_offsets is not None else ''}{M}x{N} {'fp32' if kind == 1 else 'bf16'}")
    return out if want is None or want == out.dtype else out.to(want)


def gemm_tn_two(dy, x, out, out2, accumulate: bool, expert_offsets=None, num_experts: int = 1, counts=None):
    """``[out[e]; out2[e]] (+)= dy[rows_e]ᵀ @ x[rows_e]``: the gradients of two weights that share their input, ``dy``
    holding both halves side by side.  One launch: ``x`` is read once, and twice the tiles fill the last wave."""
    R, M = dy.shape
    N = x.shape[1]
    assert dy.stride(-1) == 1 and x.stride(-1) == 1 and out.is_contiguous() and out2.is_contiguous()
    assert out.shape == out2.shape and out.dtype == out2.dtype and 2 * out.shape[-2] == M and out.shape[-1] == N
    kind = 1 if out.dtype == torch.float32 else 2
    _call("b2_gemm_tn", _p(_bf16(dy)), _p(_bf16(x)), _p(out), _p(out2), _I(M // 2), _I(M), _I(N), _I(R),
          _L(dy.stride(0)), _L(x.stride(0)), _L(N), _I(num_experts), _p(expert_offsets), _p(counts), _I(kind),
          _F(1.0 if accumulate else 0.0), _p(None), _p(status_word(dy.device)), _stream(),
          tag=f"{'grouped ' if expert_offsets is not None else ''}{M}x{N} {'fp32' if kind == 1 else 'bf16'}")


def gemm_swiglu(x, w1, w3, tile_expert=None, num_m_tiles=None, save_gate_up: bool = True, align256: bool = False):
    """``h = silu(x w1ᵀ) · (x w3ᵀ)`` per expert tile; optionally also the two pre-activations."""
    M, K = x.shape
    E, F = w1.shape[0], w1.shape[1]
    h = torch.empty(M, F, dtype=torch.bfloat16, device=x.device)
    gate = torch.empty_like(h) if save_gate_up else None
    up = torch.empty_like(h) if save_gate_up else None
    _call("b2_gemm_swiglu", _p(_bf16(x)), _p(_bf16(w1)), _p(_bf16(w3)), _p(h), _p(gate), _p(up), _I(M), _I(F), _I(K),
          _L(x.stride(0)), _I(E), _p(tile_expert), _p(num_m_tiles), _I(int(align256)), _p(status_word(x.device)),
          _stream())
    return h, gate, up


# ------------------------------------------------------------------------------ norms
def rmsnorm_fwd(x, weight, eps):
    x2 = _bf16(x).reshape(-1, x.shape[-1])
    y = torch.empty_like(x2)
    rstd = torch.empty(x2.shape[0], dtype=torch.float32, device=x.device)
    _call("b2_rmsnorm_fwd", _p(x2), _p(None), _p(weight), _p(None), _p(y), _p(rstd), _I(x2.shape[0]), _I(x2.shape[1]),
          _F(eps), _p(status_word(x.device)), _stream())
    return y.view(x.shape), rstd


def add_rmsnorm_fwd(x, delta, weight, eps):
    x2, d2 = _bf16(x).reshape(-1, x.shape[-1]), _bf16(delta).reshape(-1, x.shape[-1])
    summed, y = torch.empty_like(x2), torch.empty_like(x2)
    rstd = torch.empty(x2.shape[0], dtype=torch.float32, device=x.device)
    _call("b2_rmsnorm_fwd", _p(x2), _p(d2), _p(weight), _p(summed), _p(y), _p(rstd), _I(x2.shape[0]), _I(x2.shape[1]),
          _F(eps), _p(status_word(x.device)), _stream())
    return summed.view(x.shape), y.view(x.shape), rstd


def rmsnorm_bwd(dy, x, weight, rstd, residual_grad=None):
    x2 = x.reshape(-1, x.shape[-1])
    dy2 = _bf16(dy).reshape(-1, x.shape[-1])
    rows, D = x2.shape
    parts = require().b2_rmsnorm_bwd_parts(_I(rows), _I(D))
    partial = torch.empty(parts, D, dtype=torch.float32, device=x.device)
    dx = torch.empty_like(x2)
    dw = torch.empty(D, dtype=torch.float32, device=x.device)
    res = None if residual_grad is None else _bf16(residual_grad).reshape(-1, D).contiguous()
    _call("b2_rmsnorm_bwd", _p(dy2), _p(x2), _p(weight), _p(rstd), _p(res), _p(dx), _p(partial), _p(dw), _I(rows), _I(D),
          _p(status_word(x.device)), _stream(), n=2)
    return dx.view(x.shape), dw


# ------------------------------------------------------------------------------ router
def router_top2_fwd(logits):
    logits = logits.float().contiguous()
    T, E = logits.shape
    weights = torch.empty(T, 2, dtype=torch.float32, device=logits.device)
    idx = torch.empty(T, 2, dtype=torch.int64, device=logits.device)
    probs = torch.empty(T, E, dtype=torch.float32, device=logits.device)
    _call("b2_router_top2_fwd", _p(logits), _p(weights), _p(idx), _p(probs), _I(T), _I(E), _stream())
    return weights, idx, probs


def router_top2_bwd(dweights, probs, idx, weights):
    T, E = probs.shape
    dlogits = torch.empty(T, E, dtype=torch.float32, device=probs.device)
    _call("b2_router_top2_bwd", _p(dweights.float().contiguous()), _p(probs), _p(idx), _p(weights), _p(dlogits), _I(T),
          _I(E), _stream())
    return dlogits


def router_fwd(x, w):
    """Router product, softmax and top-2 in one launch (``w [E, D]`` bf16, E <= 16): ``(weights, idx, probs)``."""
    T, K = x.shape
    E = w.shape[0]
    probs = torch.empty(T, E, dtype=torch.float32, device=x.device)
    weights = torch.empty(T, 2, dtype=torch.float32, device=x.device)
    idx = torch.empty(T, 2, dtype=torch.int64, device=x.device)
    _call("b2_router_fwd", _p(_bf16(x)), _p(_bf16(w)), _p(weights), _p(idx), _p(probs), _I(T), _I(E), _I(K), _stream())
    return weights, idx, probs


# ------------------------------------------------------------------------------ loss
def cross_entropy_scaled_(logits, targets, loss, loss_scale: float, grad_scale: float):
    """Adds ``loss_scale · Σ_rows CE`` to ``loss`` (fp32 or fp64 scalar tensor) and overwrites ``logits`` (bf16 [T,V]) with
    ``grad_scale · (softmax − onehot)``; rows up to 32768 entries are read once and written once."""
    T, V = logits.shape
    _call("b2_cross_entropy2", _p(_bf16(logits)), _p(targets.contiguous()), _p(loss), _I(int(loss.dtype == torch.float64)), _I(T),
          _I(V), _F(loss_scale), _F(grad_scale), _p(status_word(logits.device)), _stream())
    return loss


def scale_(x, factor):
    factor = factor.to(device=x.device, dtype=torch.float32).reshape(1)
    _call("b2_scale_bf16", _p(_bf16(x)), _p(factor), _L(x.numel()), _stream())
    return x


# ------------------------------------------------------------------------------ optimizer
_DT = {torch.float32: 0, torch.bfloat16: 1}


def adamw_many_(tensors, lr, beta1, beta2, eps, weight_decay, a_t, grad_scale=1.0):
    """One update of each ``(p, g, m, v, bf16 copy of the new p or None)``; all of the same types, 48 per launch."""
    ptrs, numels = [], []
    for p, g, m, v, copy in tensors:
        if not (p.is_contiguous() and g.is_contiguous() and m.is_contiguous() and v.is_contiguous()):
            raise ValueError("adamw_ needs contiguous tensors")
        ptrs += (p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), 0 if copy is None else copy.data_ptr())
        numels.append(p.numel())
    p, g, m = tensors[0][:3]
    count = len(numels)
    _call("b2_adamw", (ctypes.c_ulonglong * (5 * count))(*ptrs), (_L * count)(*numels), _I(count), _I(_DT[p.dtype]),
          _I(_DT[g.dtype]), _I(_DT[m.dtype]), _F(lr), _F(beta1), _F(beta2), _F(eps), _F(weight_decay), _F(a_t),
          _F(grad_scale), _stream(), n=(count + 47) // 48)


def adamw_(p, g, m, v, lr, beta1, beta2, eps, weight_decay, a_t, grad_scale=1.0, p_bf16=None):
    adamw_many_([(p, g, m, v, p_bf16)], lr, beta1, beta2, eps, weight_decay, a_t, grad_scale)


def zero_many_(tensors):
    """Zeros into contiguous tensors (64 per launch).  Buffers that 16-byte stores cannot take are left to PyTorch."""
    fast = []
    for t in tensors:
        if t.is_contiguous() and t.data_ptr() % 16 == 0:
            fast.append(t)
        else:
            t.zero_()
    count = len(fast)
    if count:
        _call("b2_zero", (ctypes.c_ulonglong * count)(*[t.data_ptr() for t in fast]),
              (_L * count)(*[t.numel() * t.element_size() for t in fast]), _I(count), _stream(), n=(count + 63) // 64)


def cast_f32_bf16(src, dst):
    _call("b2_cast_f32_bf16", _p(src), _p(dst), _L(src.numel()), _stream())


# ------------------------------------------------------------------------------ embedding / rope
def embedding_fwd(ids, table):
    flat = ids.reshape(-1).contiguous()
    out = torch.empty(flat.numel(), table.shape[1], dtype=table.dtype, device=table.device)
    _call("b2_embedding_fwd", _p(flat), _p(_bf16(table)), _p(out), _I(flat.numel()), _I(table.shape[1]), _stream())
    return out.view(*ids.shape, table.shape[1])


def embedding_bwd(flat_ids, dy2d, main_grad):
    _call("b2_embedding_bwd", _p(flat_ids.contiguous()), _p(_bf16(dy2d.contiguous())), _p(main_grad),
          _I(flat_ids.numel()), _I(dy2d.shape[1]), _stream())


def _rope_table(table, seq: int, half: int):
    """A rotary table as the kernels read it: fp32, ``half`` entries for each of ``seq`` positions, 16-byte aligned."""
    if table.dtype != torch.float32 or table.numel() < seq * half:
        raise ValueError(f"rotary tables must be fp32 [>= {seq}, {half}]")
    table = table.contiguous()
    return table if table.data_ptr() % 16 == 0 else table.clone()


def rope_inplace(buf, first_elem_offset, tokens, seq, heads, head_dim, pitch, cos, sin, sign):
    cos, sin = _rope_table(cos, seq, head_dim // 2), _rope_table(sin, seq, head_dim // 2)
    ptr = ctypes.c_void_p(buf.data_ptr() + first_elem_offset * buf.element_size())
    _call("b2_rope", ptr, _p(cos), _p(sin), _I(tokens), _I(seq), _I(heads), _I(head_dim), _L(pitch), _F(sign), _stream())


# ------------------------------------------------------------------------------ device clock
def device_timestamp(out=None, index: int = 0):
    """Enqueues a one-thread kernel that stores the GPU's ``globaltimer`` (nanoseconds, one clock for the whole
    device) into ``out[index]`` (int64, allocated if not given) when the stream reaches it."""
    if out is None:
        out = torch.zeros(2, dtype=torch.int64, device=torch.device("cuda", torch.cuda.current_device()))
    _call("b2_device_timestamp", ctypes.c_void_p(out.data_ptr() + 8 * index), _stream())
    return out


# ------------------------------------------------------------------------------ all-gather fused with its GEMM
def ag_gemm_grid() -> int:
    """CTAs per launch of ``ag_gemm_nt`` (its per-block counters advance by this much per launch)."""
    return int(require().b2_ag_gemm_grid())


def ag_gemm_plan(segments, world: int, rank: int):
    """Host-only: the schedule ``ag_gemm_nt`` uses for ``rank``.  Returns ``(order, n_local, owner)``: the column
    blocks (256 rows of ``W`` each) in launch order, how many of them (the leading ones) need no peer rows, and the
    owning rank of every row.  Needs no GPU."""
    segments = [int(v) for v in segments]
    total = sum(segments)
    blocks = (total + 255) // 256
    seg = (ctypes.c_int * len(segments))(*segments)
    order = (ctypes.c_int * max(blocks, 1))()
    owner = (ctypes.c_int * max(total, 1))()
    n_local = ctypes.c_int(0)
    rc = require().b2_ag_gemm_plan(seg, _I(len(segments)), _I(world), _I(rank), _I(total), order,
                                   ctypes.byref(n_local), owner)
    if rc != 0:
        raise ValueError(f"invalid row layout for the all-gather GEMM (code {rc})")
    return list(order[:blocks]), int(n_local.value), list(owner[:total])


def ag_gemm_nt(x, w_ptrs, n_rows: int, segments, world: int, rank: int, sig_ptrs, sig_slot: int, seq: int,
               block_flags, flag_epoch: int):
    """``x [M,K] @ W [n_rows,K]ᵀ`` where ``W`` is row-sharded over ``world`` ranks: ``w_ptrs`` holds every rank's
    copy of ``W`` (a ctypes array of ``MAX_RANKS`` addresses; in copy ``r`` the rows of rank ``r`` are current).
    ``segments``: row counts of the stacked parts of ``W`` that are sharded one by one (``[n_rows]`` for a plain
    layer, ``[q, k, v]`` rows for a fused projection); inside a part of ``S`` rows rank ``r`` owns rows
    ``[r·S/world, (r+1)·S/world)``.  The kernel pulls the peers' rows into this rank's copy while the tensor cores
    work on the local rows.  ``block_flags``: int32 ``[ceil(n_rows/256)]``, zero at first use; ``flag_epoch``:
    1, 2, ... per launch with those counters.  Returns ``None`` when the device cannot co-schedule the kernel
    (gather and multiply instead)."""
    M, K = x.shape
    if x.stride(1) != 1:
        raise ValueError("x must have unit inner stride")
    segments = [int(v) for v in segments]
    if sum(segments) != n_rows:
        raise ValueError("segments must add up to the rows of W")
    seg = (ctypes.c_int * len(segments))(*segments)
    y = torch.empty(M, n_rows, dtype=torch.bfloat16, device=x.device)
    rc = require().b2_ag_gemm_nt(_p(_bf16(x)), w_ptrs, _p(y), _I(M), _I(n_rows), _I(K), _L(x.stride(0)), _L(n_rows),
                                 seg, _I(len(segments)), _I(world), _I(rank), sig_ptrs, _I(sig_slot), _I(seq),
                                 _p(block_flags), _I(flag_epoch), _p(status_word(x.device)), _stream())
    if rc == -20:
        return None
    if rc != 0:
        raise RuntimeError(f"b2_ag_gemm_nt failed with code {rc}")
    global _launches
    _launches += 1
    return y


# ------------------------------------------------------------------------------ attention
def _token_pitch(t):
    B, S, H, hd = t.shape
    if hd != 128 or t.stride(3) != 1 or t.stride(2) != hd or t.stride(0) != S * t.stride(1):
        raise ValueError("attention tensors must be [B, S, H, 128] views with contiguous heads and uniform token pitch")
    return t.stride(1)


def _pitched(t) -> bool:
    """``[B, S, H, 128]`` with contiguous heads, one token pitch throughout, and the alignment that 16-byte vectors and
    tensor maps need."""
    S, H, hd = t.shape[1:]
    return (hd == 128 and t.stride(3) == 1 and t.stride(2) == hd and t.stride(0) == S * t.stride(1)
            and t.stride(1) >= H * hd and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0)


def attention_fwd(q, k, v, cos=None, sin=None, causal=True):
    """GQA attention, causal by default.  ``q [B,S,Hq,128]``, ``k, v [B,S,Hkv,128]`` bf16 (views of a fused projection are
    fine), or all three fp16 without a rotation; any ``S``.  With ``cos``/``sin`` (fp32 ``[>= S, 64]``) rotated copies of
    q and k are made first.  Returns ``(out [B,S,Hq,128], lse fp32 [B,Hq,S], q_used, k_used)``."""
    B, S, Hq, hd = q.shape
    Hkv = k.shape[2]
    f16 = q.dtype == k.dtype == v.dtype == torch.float16 and cos is None
    if cos is not None:
        cos, sin = _rope_table(cos, S, 64), _rope_table(sin, S, 64)
        q, k = (t if _pitched(_bf16(t)) else t.clone(memory_format=torch.contiguous_format) for t in (q, k))
        qr, kr = (torch.empty(t.shape, dtype=torch.bfloat16, device=t.device) for t in (q, k))
        _call("b2_rope_copy", _p(q), _p(k), _p(qr), _p(kr), _p(cos), _p(sin), _I(B * S), _I(S), _I(Hq), _I(Hkv),
              _L(_token_pitch(q)), _L(_token_pitch(k)), _stream())
        q, k = qr, kr
    if not f16:
        _bf16(q), _bf16(k), _bf16(v)
    out = torch.empty(B, S, Hq, hd, dtype=q.dtype, device=q.device)
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device=q.device)
    _call("b2_attention_fwd_ex", _p(q), _p(k), _p(v), _L(_token_pitch(q)), _L(_token_pitch(k)),
          _L(_token_pitch(v)), _p(out), _p(lse), _I(B), _I(S), _I(Hq), _I(Hkv), _F(hd ** -0.5), _I(int(causal)),
          _I(int(f16)), _p(status_word(q.device)), _stream())
    return out, lse, q, k


def attention_bwd(dout, q, k, v, out, lse, cos=None, sin=None, grads=None, causal=True):
    """Gradients of ``attention_fwd``.  ``q`` and ``k`` are the tensors the forward kernel saw (rotated, if a
    rotation was applied); with ``cos``/``sin`` the kernels store dq and dk rotated back, i.e. as gradients of the
    unrotated q and k.  ``grads`` may give three preallocated ``[B,S,H,128]`` views (for instance slices of one
    fused buffer) to write into."""
    B, S, Hq, hd = q.shape
    Hkv = k.shape[2]
    if grads is None:
        grads = (torch.empty(B, S, Hq, hd, dtype=torch.bfloat16, device=q.device),
                 torch.empty(B, S, Hkv, hd, dtype=torch.bfloat16, device=q.device),
                 torch.empty(B, S, Hkv, hd, dtype=torch.bfloat16, device=q.device))
    dq, dk, dv = grads
    # per query row -lse*log2(e) and -rowsum(dO*O), rows padded to whole tiles
    stats = torch.empty(B * Hq, 2, (S + 127) // 128 * 128, dtype=torch.float32, device=q.device)
    dout = _bf16(dout).contiguous()
    if cos is not None and (cos.shape[-1] != 64 or not cos.is_contiguous() or cos.shape[0] < S):
        raise ValueError("rotary tables must be contiguous fp32 [>= S, 64]")
    _call("b2_attention_bwd_rope", _p(dout), _p(q), _p(k), _p(v), _p(_bf16(out)), _p(lse), _L(_token_pitch(q)),
          _L(_token_pitch(k)), _L(_token_pitch(v)), _p(stats), _p(dq), _p(dk), _p(dv), _L(_token_pitch(dq)),
          _L(_token_pitch(dk)), _L(_token_pitch(dv)), _I(B), _I(S), _I(Hq), _I(Hkv), _F(hd ** -0.5),
          _I(int(causal)), _p(cos), _p(sin), _p(status_word(q.device)), _stream(), n=3)
    return dq, dk, dv


# ------------------------------------------------------------------------------ MoE routing
def moe_plan(idx, num_experts, capacity_rows):
    slots = idx.numel()
    dev = idx.device
    # one allocation, cut into the six tables (the kernel writes what it promises of each)
    sizes = (slots, capacity_rows, num_experts, capacity_rows // 128, 4, num_experts)
    slot_row, row_slot, offs, tile_expert, meta, counts = torch.empty(sum(sizes), dtype=torch.int32,
                                                                      device=dev).split(sizes)
    _call("b2_moe_plan", _p(idx.contiguous()), _I(slots), _I(num_experts), _p(slot_row), _p(row_slot), _p(offs),
          _p(tile_expert), _p(meta), _p(counts), _I(capacity_rows), _stream())
    return slot_row, row_slot, offs, tile_expert, meta, counts


def moe_gather(x, row_slot, meta, capacity_rows, scale=None, y_perm=None, dweights=None, out=None):
    D = x.shape[1]
    if out is None:
        out = torch.empty(capacity_rows, D, dtype=torch.bfloat16, device=x.device)
    _call("b2_moe_gather", _p(_bf16(x)), _p(row_slot), _p(meta), _p(scale), _p(y_perm), _p(dweights), _p(out), _I(D),
          _I(capacity_rows), _I(2 * x.shape[0]), _stream())
    return out


def moe_combine(y_perm, slot_row, weights, tokens, residual=None):
    D = y_perm.shape[1]
    out = torch.empty(tokens, D, dtype=torch.bfloat16, device=y_perm.device)
    _call("b2_moe_combine", _p(_bf16(y_perm)), _p(slot_row), _p(weights), _p(residual), _p(out), _I(tokens), _I(D),
          _I(y_perm.shape[0]), _stream())
    return out


def moe_aux(probs, counts):
    """Balance loss of top-2 routing from the router's probabilities ``[T, E]`` and the experts' slot counts."""
    aux = torch.empty((), dtype=torch.float32, device=probs.device)
    _call("b2_moe_aux", _p(probs), _p(counts), _p(aux), _I(probs.shape[0]), _I(probs.shape[1]), _stream())
    return aux


def moe_dx(dy_perm, slot_row, dweights, probs, idx, weights, router_w, daux=None, counts=None):
    """Input gradient of a routed layer: the two rows of each token plus the router's share, that of the balance loss
    (``daux``: its gradient, fp32 device scalar) included; returns ``(dx, dlogits)``."""
    T, E = probs.shape
    D = dy_perm.shape[1]
    dlogits = torch.empty(T, E, dtype=torch.float32, device=dy_perm.device)
    dx = torch.empty(T, D, dtype=torch.bfloat16, device=dy_perm.device)
    _call("b2_moe_dx", _p(_bf16(dy_perm)), _p(slot_row), _p(dweights), _p(probs), _p(idx), _p(weights), _p(daux), _p(counts),
          _p(_bf16(router_w)), _p(dlogits), _p(dx), _I(T), _I(E), _I(D), _I(dy_perm.shape[0]), _stream())
    return dx, dlogits


def swiglu_bwd(dh, gate, up, live_rows=None, want_h: bool = True):
    rows, F = dh.shape
    dgu = torch.empty(rows, 2 * F, dtype=torch.bfloat16, device=dh.device)
    h = torch.empty(rows, F, dtype=torch.bfloat16, device=dh.device) if want_h else None
    _call("b2_swiglu_bwd", _p(_bf16(dh)), _p(gate), _p(up), _p(dgu), _p(h), _p(live_rows), _I(rows), _I(F), _stream())
    return dgu, h


# ------------------------------------------------------------------------------ expert-parallel return in the epilogue
def gemm_nt_push(a, w, tile_expert, num_m_tiles, num_experts, dst_table, row_tag, row_src, row_w, sig_table,
                 sig_slot: int, seq: int, rank: int, n: int, ticket):
    """Rows of ``a [M,K] @ w[e] [N,K]ᵀ``, scaled by ``row_w`` (or 1), stored as bf16 into row ``row_tag[r]`` of rank
    ``row_src[r]``'s buffer (``dst_table``: ctypes array of ``MAX_RANKS`` addresses, row pitch ``N``); afterwards
    flag ``seq`` is raised in slot ``sig_slot`` of every rank's signal pad."""
    M, K = a.shape
    N = w.shape[-2]
    assert a.stride(-1) == 1 and w.is_contiguous()
    _call("b2_gemm_nt_push", _p(_bf16(a)), _p(_bf16(w)), _I(M), _I(N), _I(K), _L(a.stride(0)), _I(num_experts),
          _p(tile_expert), _p(num_m_tiles), _I(1), dst_table, _p(row_tag), _p(row_src), _p(row_w), sig_table,
          _I(sig_slot), _I(seq), _I(rank), _I(n), _p(ticket), _p(status_word(a.device)), _stream())


def gemm_nn_push(a, w, w2, tile_expert, num_m_tiles, num_experts, dst_table, row_tag, row_src, row_w, sig_table,
                 sig_slot: int, seq: int, rank: int, n: int, ticket):
    """The same for ``a [M,K] @ [w[e]; w2[e]]`` (``w``, ``w2``: ``[E, K/2, N]``, the reduction runs over their rows)."""
    M, K = a.shape
    N = w.shape[-1]
    k_split = w.shape[-2] if w2 is not None else 0
    assert a.stride(-1) == 1 and w.is_contiguous()
    _call("b2_gemm_nn_push", _p(_bf16(a)), _p(_bf16(w)), _p(w2), _I(M), _I(N), _I(K), _I(k_split), _L(a.stride(0)),
          _I(num_experts), _p(tile_expert), _p(num_m_tiles), _I(1), dst_table, _p(row_tag), _p(row_src), _p(row_w),
          sig_table, _I(sig_slot), _I(seq), _I(rank), _I(n), _p(ticket), _p(status_word(a.device)), _stream())


def ep_swiglu_bwd(dh, gate_lo, up_lo, gate_hi, up_hi, split_row: int, dgu, meta, row_tag, row_src, row_w,
                  dw_table, n: int):
    """SwiGLU backward on expert-major rows with the routing weight folded in (see ``ep_swiglu_bwd_kernel``):
    ``dh`` is overwritten with ``w·h``, ``dgu`` receives ``w·[dgate | dup]``, the routing-weight gradient of every
    row goes to its source rank's ``dw_table`` entry."""
    rows, F = dh.shape
    _call("b2_ep_swiglu_bwd", _p(_bf16(dh)), _p(gate_lo), _p(up_lo), _p(gate_hi), _p(up_hi), _I(split_row), _p(dgu),
          _p(meta), _p(row_tag), _p(row_src), _p(row_w), dw_table, _I(rows), _I(F), _I(n), _stream())
