"""sm_100a kernels against plain PyTorch fp32 statements of the same ops."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def native():
    from b200moe.ops import native as n
    n.require()
    return n


@pytest.fixture(params=[0, 2, 3], ids=["tiles_auto", "tiles_256_one_cta", "tiles_cta_pair"])
def tile_mode(request, native):
    """GEMM CTA tile: automatic choice, forced single-CTA 256x256, forced CTA pairs (cta_group::2)."""
    native.set_gemm_tile_mode(request.param)
    yield request.param
    native.set_gemm_tile_mode(0)


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).bfloat16()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (384, 1024, 4096), (1024, 6144, 1024),
                                   (200, 384, 192), (128, 32000, 512)])
def test_gemm_nt(native, tile_mode, M, N, K):
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    got = native.gemm_nt(x, w)
    want = x.float() @ w.float().t()
    assert _rel(got, want) < 6e-3
    native.check_status()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 1024, 512), (384, 4096, 2048), (256, 320, 128)])
def test_gemm_nn(native, tile_mode, M, N, K):
    dy, w = _rand(M, K), _rand(K, N, scale=0.05)
    got = native.gemm_nn(dy, w)
    assert _rel(got, dy.float() @ w.float()) < 6e-3
    native.check_status()


@pytest.mark.parametrize("R,M,N", [(128, 128, 256), (512, 256, 512), (4096, 1024, 384), (1024, 6144, 1024)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gemm_tn_accumulates(native, tile_mode, R, M, N, dtype):
    dy, x = _rand(R, M, scale=0.1), _rand(R, N, scale=0.1)
    base = torch.randn(M, N, device="cuda").to(dtype)
    out = base.clone()
    native.gemm_tn(dy, x, out=out, accumulate=True)
    want = base.float() + dy.float().t() @ x.float()
    assert _rel(out, want) < (2e-3 if dtype == torch.float32 else 8e-3)
    fresh = native.gemm_tn(dy, x, out_dtype=torch.float32)
    assert _rel(fresh, dy.float().t() @ x.float()) < 2e-3
    native.check_status()


def test_fp32_additions_keep_subnormals_and_round_the_scaled_product(native, tile_mode):
    """What the memory system adds is what the SM would add: exact with subnormal terms and sums; with a factor the product is
    rounded, then added."""
    for old, left, right in ((1e-39, 0.0, 0.0), (0.0, 2.0 ** -70, 2.0 ** -63), (2.0 ** -126, 2.0 ** -70, 2.0 ** -63),
                             (-2.0 ** -126, 2.0 ** -65, 2.0 ** -62)):
        dy, x = (torch.zeros(64, n, device="cuda").bfloat16() for n in (136, 96))
        dy[5], x[5] = left, right
        got = torch.full((136, 96), old, device="cuda")
        want = float(got[0, 0].double()) + left * right             # a sum that fp32 holds
        native.gemm_tn(dy, x, out=got, accumulate=True)
        assert bool((got.double() == want).all())
    dy, x, factor, old = _rand(100, 136), _rand(100, 96), torch.tensor(0.3, device="cuda"), torch.randn(136, 96, device="cuda")
    want = native.gemm_tn(dy, x) * factor + old
    native.gemm_tn(dy, x, out=old, accumulate=True, alpha=factor)
    assert torch.equal(old, want)
    native.check_status()


@pytest.mark.parametrize("M,N,K", [(1, 2112, 64), (15, 4096, 4096), (16, 4096, 4096), (7, 9472, 512)])
def test_products_of_few_rows(native, M, N, K):
    """An A operand below 128 KiB, where 64 columns per tile would make many CTAs, and the first one that is not."""
    x, w = _rand(M, K), _rand(N, K, scale=K ** -0.5)
    got = native.gemm_nt(x, w)
    want = x.double() @ w.double().t()
    # bf16 result: half an ulp, beside K additions of 2^-24
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())).all())
    native.set_gemm_tile_mode(1)
    assert torch.equal(native.gemm_nt(x, w), got) and torch.equal(native.gemm_nn(x, w.t().contiguous()), got)
    native.set_gemm_tile_mode(0)
    assert torch.equal(native.gemm_nn(x, w.t().contiguous()), got)
    native.check_status()


@pytest.mark.parametrize("mode", [6, 7], ids=["128x128", "128x64"])
@pytest.mark.parametrize("M,N,K", [(1, 32, 64), (129, 96, 128), (200, 320, 576), (300, 2080, 64), (2100, 1312, 192)])
def test_narrow_tiles_give_the_bits_of_wide_ones(native, mode, M, N, K):
    """Every product on tiles of 128 and 64 columns (rows and columns behind the last tile; one tile, several waves): each
    element is the same chain of additions as on 128x256 tiles."""
    x, w, wt = _rand(M, K), _rand(N, K, scale=0.1), _rand(K, N, scale=0.1)
    F = 128 * (N // 128 + 1)
    w1, w3 = _rand(1, F, K, scale=0.1), _rand(1, F, K, scale=0.1)
    gate, up, left, right = _rand(M, N), _rand(M, N), _rand(K, 8 * (M // 8 + 1)), _rand(K, N)
    base = torch.randn(left.shape[1], N, device="cuda")
    cos, sin = torch.rand(M, 64, device="cuda"), torch.rand(M, 64, device="cuda")
    half = torch.full((), 0.375, device="cuda")

    def products():
        sums = [base.clone(), base.bfloat16()]
        for out in sums:
            native.gemm_tn(left, right, out=out, accumulate=True, alpha=half)
        return [native.gemm_nt(x, w), native.gemm_nt(x, w, out_dtype=torch.float32),
                native.gemm_nt_rope(x, w, cos, sin, N // 128 * 128, M), native.gemm_nn(x, wt, alpha=half),
                native.gemm_nn(torch.cat((x, x), 1), wt, w2=wt), *native.gemm_swiglu(x, w1, w3),
                *(native.gemm_nn_swiglu_bwd(x, wt, gate, up) if M * N <= 1 << 21 else ()), *sums,
                native.gemm_tn(left, right, out_dtype=torch.bfloat16)]

    try:
        native.set_gemm_tile_mode(1)
        want = products()
        native.set_gemm_tile_mode(mode)
        got = products()
    finally:
        native.set_gemm_tile_mode(0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert _rel(got[0], x.float() @ w.float().t()) < 6e-3
    native.check_status()


@pytest.mark.parametrize("mode", [6, 7], ids=["128x128", "128x64"])
@pytest.mark.parametrize("counts", [[100, 0, 300, 17], [256, 1, 64, 65]])
def test_grouped_products_on_narrow_tiles(native, mode, counts):
    offs, tile_expert, meta, rows = _segments(counts, 256)
    E, D, F = len(counts), 192, 384
    x, dy = torch.zeros(rows, D, device="cuda").bfloat16(), torch.zeros(rows, F, device="cuda").bfloat16()
    for e, n in enumerate(counts):
        lo = 0 if e == 0 else int(offs[e - 1])
        x[lo:lo + n], dy[lo:lo + n] = _rand(n, D), _rand(n, F)
    w1, w3, w2 = _rand(E, F, D, scale=0.1), _rand(E, F, D, scale=0.1), _rand(E, D, F, scale=0.1)
    count, base = torch.tensor(counts, device="cuda", dtype=torch.int32), torch.randn(E, F, D, device="cuda")

    def products():
        h, gate, up = native.gemm_swiglu(x, w1, w3, tile_expert, meta[:1], align256=True)
        out = native.gemm_nt(h, w2, tile_expert=tile_expert, num_m_tiles=meta[:1], num_experts=E, align256=True)
        dx = native.gemm_nn(dy, w1, tile_expert=tile_expert, num_m_tiles=meta[:1], num_experts=E, align256=True)
        dw = native.gemm_tn(dy, x, out=base.clone(), accumulate=True, expert_offsets=offs, num_experts=E, counts=count)
        return h, gate, up, out, dx, dw

    try:
        native.set_gemm_tile_mode(1)
        want = products()
        native.set_gemm_tile_mode(mode)
        got = products()
    finally:
        native.set_gemm_tile_mode(0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    native.check_status()


@pytest.mark.parametrize("R,F,N", [(64, 4, 32), (100, 36, 96), (129, 264, 288)])
@pytest.mark.parametrize("accumulate", [True, False])
def test_fp32_results_cut_between_two_weights(native, tile_mode, R, F, N, accumulate):
    """The bulk stores of fp32 results: rows behind the matrix, and a cut that lies inside a warp's 32 rows."""
    dy, x = _rand(R, 2 * F, scale=0.1), _rand(R, N, scale=0.1)
    guard = torch.randn(3, F, N, device="cuda")
    got = guard.clone()
    native.gemm_tn_two(dy, x, got[0], got[1], accumulate)
    product = (dy.double().t() @ x.double()).view(2, F, N)
    want = product + guard[:2].double() if accumulate else product
    # products of bf16 are exact in fp32; R additions and the final one round to 2^-24 of the running sum each
    bound = (R + 1) * 2.0 ** -24 * (dy.double().abs().t() @ x.double().abs()).view(2, F, N) + 2.0 ** -24 * guard[:2].abs()
    assert bool(((got[:2].double() - want).abs() <= bound * 1.01 + 1e-30).all())
    assert torch.equal(got[2], guard[2])
    native.check_status()


def _segments(counts, pad=128):
    padded = [(c + pad - 1) // pad * pad for c in counts]
    offs, tiles, row = [], [], 0
    for e, p in enumerate(padded):
        tiles += [e] * (p // 128)
        row += p
        offs.append(row)
    dev = dict(device="cuda", dtype=torch.int32)
    return (torch.tensor(offs, **dev), torch.tensor(tiles, **dev), torch.tensor([len(tiles), row, 0, 0], **dev), row)


@pytest.mark.parametrize("R,M,N", [(64, 8, 32), (100, 136, 96), (129, 264, 288), (64, 520, 352)])
def test_bf16_products_are_the_fp32_ones_rounded_once(native, tile_mode, R, M, N):
    """Columns that end inside the 64 of a staged row, rows that end inside a warp's 32: bit for bit the fp32 result
    of the same tiles, rounded; with a factor, and cut into two outputs."""
    dy, x, alpha = _rand(R, M), _rand(R, N), torch.tensor(0.37, device="cuda")
    exact = native.gemm_tn(dy, x, out_dtype=torch.float32, alpha=alpha)
    assert torch.equal(native.gemm_tn(dy, x, out_dtype=torch.bfloat16, alpha=alpha), exact.bfloat16())
    halves = [torch.empty(1, M // 2, N, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    native.gemm_tn_two(dy, x, *halves, False)
    whole = native.gemm_tn(dy, x, out_dtype=torch.float32, alpha=torch.ones((), device="cuda"))
    assert torch.equal(torch.cat(halves, 1)[0], whole.view(M, N).bfloat16())
    native.check_status()


@pytest.mark.parametrize("pad", [128, 256])
@pytest.mark.parametrize("counts", [[128, 256], [100, 0, 300, 17], [0, 0, 640, 0], [384] * 4])
def test_grouped_expert_gemms(native, tile_mode, counts, pad):
    """``pad`` = 256: expert segments are whole 256-row tiles, which makes the 256-row tile kinds legal."""
    torch.manual_seed(0)
    E, D, Fd = len(counts), 256, 512
    offs, tile_expert, meta, rows = _segments(counts, pad)
    align = pad == 256
    cap = rows + 256                                  # rows past the live count must be ignored
    x = torch.zeros(cap, D, device="cuda", dtype=torch.bfloat16)
    start = 0
    for e, c in enumerate(counts):
        x[start:start + c] = _rand(c, D)
        start = int(offs[e])
    x[rows:] = float("nan")
    w1, w3, w2 = _rand(E, Fd, D, scale=0.05), _rand(E, Fd, D, scale=0.05), _rand(E, D, Fd, scale=0.05)
    h, gate, up = native.gemm_swiglu(x, w1, w3, tile_expert, meta[0:1], align256=align)
    y = native.gemm_nt(h, w2, tile_expert=tile_expert, num_m_tiles=meta[0:1], num_experts=E, align256=align)
    start = 0
    for e in range(E):
        end = int(offs[e])
        if end > start:
            xe = x[start:end].float()
            g, u = xe @ w1[e].float().t(), xe @ w3[e].float().t()
            he = torch.nn.functional.silu(g) * u
            assert _rel(gate[start:end], g) < 6e-3 and _rel(up[start:end], u) < 6e-3
            assert _rel(h[start:end], he) < 8e-3
            assert _rel(y[start:end], h[start:end].float() @ w2[e].float().t()) < 6e-3
        start = end
    # data gradients: dh = dy W2 ; dx = dg W1 + du W3 in one pass
    dy = torch.zeros(cap, D, device="cuda", dtype=torch.bfloat16)
    dy[:rows] = _rand(rows, D)
    dh = native.gemm_nn(dy, w2, tile_expert=tile_expert, num_m_tiles=meta[0:1], num_experts=E, align256=align)
    dgu = torch.zeros(cap, 2 * Fd, device="cuda", dtype=torch.bfloat16)
    dgu[:rows] = _rand(rows, 2 * Fd, scale=0.1)
    dx = native.gemm_nn(dgu, w1, w2=w3, tile_expert=tile_expert, num_m_tiles=meta[0:1], num_experts=E,
                        align256=align)
    acc = torch.randn(E, Fd, D, device="cuda")
    dw1 = acc.clone()
    native.gemm_tn(dgu[:, :Fd], x, out=dw1, accumulate=True, expert_offsets=offs, num_experts=E)
    dw_new = native.gemm_tn(dy, h, out_dtype=torch.float32, expert_offsets=offs, num_experts=E)
    start = 0
    for e in range(E):
        end = int(offs[e])
        if end > start:
            assert _rel(dh[start:end], dy[start:end].float() @ w2[e].float()) < 6e-3
            want = dgu[start:end, :Fd].float() @ w1[e].float() + dgu[start:end, Fd:].float() @ w3[e].float()
            assert _rel(dx[start:end], want) < 6e-3
            assert _rel(dw1[e], acc[e] + dgu[start:end, :Fd].float().t() @ x[start:end].float()) < 3e-3
            assert _rel(dw_new[e], dy[start:end].float().t() @ h[start:end].float()) < 3e-3
        else:
            assert torch.equal(dw1[e], acc[e]) and float(dw_new[e].abs().max()) == 0.0
        start = end
    native.check_status()


@pytest.mark.parametrize("tokens,dim,ffn,launches", [(1, 64, 128, 6), (129, 192, 384, 6), (300, 512, 640, 6),
                                                     (5500, 64, 384, 7)])
def test_dense_swiglu_layer_on_the_fused_kernels(native, tile_mode, tokens, dim, ffn, launches):
    """Rows and widths around the tile edges, in every tile kind, forward and all gradients against 64 bits; a hook on
    one projection sends the same layer through the three separate products."""
    from b200moe.models.layers import PositionWiseFFLayer
    torch.manual_seed(tokens)
    layer = PositionWiseFFLayer(dim, ffn, device="cuda").to(torch.bfloat16)
    x = _rand(tokens, dim).requires_grad_(True)
    dy = _rand(tokens, dim)
    leaves = [t.detach().double().requires_grad_(True) for t in (x, layer.w1.weight, layer.w3.weight, layer.w2.weight)]
    gate = leaves[0] @ leaves[1].t()
    ref = (gate * torch.sigmoid(gate) * (leaves[0] @ leaves[2].t())) @ leaves[3].t()
    wanted = torch.autograd.grad(ref, leaves, dy.double())
    calls = []
    for hook in (False, True):
        if hook:
            layer.w3.register_forward_hook(lambda *_: calls.append(1))
        for p in (x, *layer.parameters()):
            p.grad = None
        before = native.launch_count()
        out = layer(x)
        out.backward(dy)
        assert native.launch_count() - before == (9 if hook else launches)
        # bf16 hidden layer and gradients of it: 2^-9 each, three roundings deep
        assert _rel(out, ref) < 1e-2
        for got, want in zip((x.grad, layer.w1.weight.grad, layer.w3.weight.grad, layer.w2.weight.grad), wanted):
            assert _rel(got, want) < 1.2e-2
    assert calls
    native.check_status()


@pytest.mark.parametrize("counts", [[100, 0, 300, 17], [256, 1, 64, 65], [0, 0, 640, 0]])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_grouped_weight_gradients_of_two_weights_over_live_rows(native, tile_mode, counts, dtype):
    """Two accumulators from one launch (their border inside a 256-row tile), the reduction cut at each expert's count:
    what lies in the padding behind the last started 64 rows is not read."""
    torch.manual_seed(1)
    E, F, D = len(counts), 160, 96
    offs, _, _, rows = _segments(counts, 256)
    dy, x = _rand(rows, 2 * F, scale=0.1), _rand(rows, D, scale=0.1)
    start, live = 0, torch.zeros(rows, dtype=torch.bool, device="cuda")
    for e, c in enumerate(counts):
        end = int(offs[e])
        live[start:start + c] = True
        dy[start + c:end] = 0
        x[start + c:end] = 0
        x[min(start + (c + 63) // 64 * 64, end):end] = float("nan")
        start = end
    base = [torch.randn(E, F, D, device="cuda").to(dtype) for _ in range(2)]
    got = [t.clone() for t in base]
    count = torch.tensor(counts, dtype=torch.int32, device="cuda")
    native.gemm_tn_two(dy, x, *got, True, offs, E, count)
    third = native.gemm_tn(dy[:, :F], x, out=base[0].clone(), accumulate=True, expert_offsets=offs, num_experts=E, counts=count)
    assert torch.equal(third, got[0])
    start = 0
    for e, c in enumerate(counts):
        want = dy[start:start + c].double().t() @ x[start:start + c].double()
        for half in range(2):
            assert _rel(got[half][e].double(), base[half][e].double() + want[half * F:(half + 1) * F]) < (
                1e-5 if dtype == torch.float32 else 4e-3)
        start = int(offs[e])
    native.check_status()


def test_rmsnorm_forward_backward(native):
    from b200moe import ops
    from b200moe.ops import functional as Fn
    for D in (128, 4096):
        x = _rand(300, D).requires_grad_(True)
        d = _rand(300, D).requires_grad_(True)
        w = (torch.rand(D, device="cuda") + 0.5).requires_grad_(True)
        y = ops.rmsnorm(x, w)
        xr, wr = x.detach().float().requires_grad_(True), w.detach().clone().requires_grad_(True)
        yr = Fn.rmsnorm_ref(xr, wr)
        assert _rel(y, yr) < 5e-3
        dy = _rand(300, D)
        y.backward(dy)
        yr.backward(dy.float())
        assert _rel(x.grad, xr.grad) < 8e-3 and _rel(w.grad, wr.grad) < 8e-3
        x.grad = w.grad = None
        s, y2 = ops.add_rmsnorm(x, d, w)
        (s.float().sum() * 0.5 + (y2.float() * dy.float()).sum()).backward()
        xs = (x.detach().float() + d.detach().float()).bfloat16().float().requires_grad_(True)
        wr2 = w.detach().clone().requires_grad_(True)
        (xs.sum() * 0.5 + (Fn.rmsnorm_ref(xs, wr2) * dy.float()).sum()).backward()
        assert _rel(s, xs) < 1e-6 and _rel(x.grad, xs.grad) < 8e-3 and _rel(d.grad, xs.grad) < 8e-3
        assert _rel(w.grad, wr2.grad) < 8e-3


@pytest.mark.parametrize("rows,D", [(1, 8), (3563, 512), (1800, 520), (1777, 1024), (893, 2048), (451, 2056), (450, 8192),
                                    (65, 512), (2368, 512), (2369, 512), (592, 2048), (148, 8192), (149, 4104)])
def test_rmsnorm_row_blocks(native, rows, D):
    """Blocks of eight to one rows through the ring, the last one cut short; the one-CTA-per-row form of few rows; backward
    without the ring where no CTA has a second block."""
    x, delta, dy, res = (_rand(rows, D) for _ in range(4))
    w = torch.rand(D, device="cuda") + 0.5
    summed, y, rstd = native.add_rmsnorm_fwd(x, delta, w, 1e-5)
    few = native.add_rmsnorm_fwd(x[-3:], delta[-3:], w, 1e-5)
    assert all(torch.equal(a[-3:], b) for a, b in zip((summed, y, rstd), few))
    assert torch.equal(summed, (x.float() + delta.float()).bfloat16())
    s64, w64, dy64 = summed.double(), w.double(), dy.double()
    r64 = (s64.square().mean(1) + 1e-5).rsqrt()
    # rstd: D additions and a few operations in fp32; y: one more rounding to bf16
    assert bool(((rstd.double() / r64 - 1).abs() <= (D + 8) * 2.0 ** -24).all())
    assert bool(((y.double() - s64 * r64[:, None] * w64).abs() <= 2.0 ** -8 * (s64 * r64[:, None] * w64).abs() + 1e-30).all())
    for residual in (None, res):
        dx, dw = native.rmsnorm_bwd(dy, summed, w, rstd, residual_grad=residual)
        xhat, g = s64 * r64[:, None], dy64 * w64
        want = r64[:, None] * (g - xhat * (g * xhat).mean(1, keepdim=True)) + (0 if residual is None else residual.double())
        assert _rel(dx, want) < 4e-3
        bound = (rows + 8) * 2.0 ** -23 * (dy64 * xhat).abs().sum(0)
        assert bool(((dw.double() - (dy64 * xhat).sum(0)).abs() <= bound + 1e-30).all())
        if rows > 1:                              # rows do not depend on how many there are, ring or not
            assert torch.equal(native.rmsnorm_bwd(dy[-1:], summed[-1:], w, rstd[-1:], None if residual is None else res[-1:])[0], dx[-1:])
    native.check_status()


@pytest.mark.parametrize("T,D", [(64, 128), (300, 512), (2048, 1024)])
def test_launches_that_overlap_keep_their_order(native, T, D):
    """Kernels are placed while the one before them still runs: reads and writes of shared buffers, one after the other,
    replayed from a graph and on a second stream, give the bits of a run that waits for every kernel."""
    ids = torch.randint(0, 50, (T,), device="cuda")
    table, w, w2 = _rand(50, D), _rand(2 * D, D, scale=D ** -0.5), _rand(2 * D, D, scale=(2 * D) ** -0.5)
    gain = torch.rand(D, device="cuda") + 0.5
    x, y = _rand(T, D), torch.empty(T, D, device="cuda").bfloat16()
    acc = torch.zeros(2 * D, D, device="cuda")

    def run(wait):
        wait()
        native.zero_many_([acc])
        wait()
        cur = native.embedding_fwd(ids, table)
        for _ in range(6):
            wait()
            summed, normed, rstd = native.add_rmsnorm_fwd(cur, x, gain, 1e-5)
            wait()
            up = native.gemm_nt(normed, w)
            wait()
            native.gemm_nn(up, w2, out=y)
            wait()
            native.gemm_tn(up, normed, out=acc, accumulate=True)
            wait()
            cur, dgain = native.rmsnorm_bwd(y, summed, gain, rstd)
        wait()
        return torch.cat((cur.float().flatten(), acc.flatten(), dgain))

    want = run(torch.cuda.synchronize)
    none = lambda: None  # noqa: E731
    assert all(torch.equal(run(none), want) for _ in range(5))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = run(none)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(other, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run(none)
    for _ in range(3):
        graph.replay()
        assert torch.equal(captured, want)
    native.check_status()


@pytest.mark.parametrize("T,S", [(256, 128), (2048, 1024)])
def test_overlapping_launches_of_routing_attention_loss_and_optimizer(native, T, S):
    """The same for the kernels of a block around the products (from 1280 tokens on the plan is a cluster's, 1024 tokens a sequence
    share backward steps between CTAs), with PyTorch operations in between."""
    D, F_, E, V = 512, 256, 4, 320
    cap = (2 * T + E * 255 + 255) // 256 * 256
    x0, router = _rand(T, D), _rand(E, D, scale=D ** -0.5)
    w1, w3, w2 = _rand(E, F_, D, scale=D ** -0.5), _rand(E, F_, D, scale=D ** -0.5), _rand(E, D, F_, scale=F_ ** -0.5)
    head, targets = _rand(V, D, scale=D ** -0.5), torch.randint(0, V, (T,), device="cuda")
    m, v = torch.zeros(V, D, device="cuda"), torch.zeros(V, D, device="cuda")
    acc, master = torch.zeros(V, D, device="cuda"), torch.zeros(V, D, device="cuda")

    def run(wait):
        def after(value):
            wait()
            return value

        native.zero_many_([acc, m, v, master])
        x = after(x0 * 1)
        for _ in range(3):
            weights, idx, probs = after(native.router_fwd(x, router))
            slot_row, row_slot, offs, tiles, meta, counts = after(native.moe_plan(idx, E, cap))
            rows = after(native.moe_gather(x, row_slot, meta, cap))
            h, gate, up = after(native.gemm_swiglu(rows, w1, w3, tiles, meta[:1], align256=True))
            y = after(native.gemm_nt(h, w2, tile_expert=tiles, num_m_tiles=meta[:1], num_experts=E, align256=True))
            x = after(native.moe_combine(y, slot_row, weights, T, residual=x))
            aux = after(native.moe_aux(probs, counts))
            dweights = torch.empty(T, 2, device="cuda")
            dy = after(native.moe_gather(x, row_slot, meta, cap, scale=weights.view(-1), y_perm=y, dweights=dweights.view(-1)))
            dx, dlogits = after(native.moe_dx(dy, slot_row, dweights, probs, idx, weights, router, aux, counts))
            q = after((x + dx).view(T // S, S, 4, 128).clamp(-4, 4))
            out, lse, _, _ = after(native.attention_fwd(q, q, q))
            grads = after(native.attention_bwd(q, q, q, q, out, lse))
            x = after(sum(grads).clamp(-4, 4).reshape(T, D))
            logits = after(native.gemm_nt(x, head))
            loss = after(native.cross_entropy_scaled_(logits, targets, torch.zeros((), dtype=torch.float64, device="cuda"), 1 / T, 1.0))
            after(native.gemm_tn(logits, x, out=acc, accumulate=True))
            after(native.adamw_(master, acc, m, v, 1e-3, 0.9, 0.999, 1e-8, 0.0, 1e-3))
        wait()
        return torch.cat([t.float().flatten() for t in (x, dlogits, loss, acc, master, m, v)])

    want = run(torch.cuda.synchronize)
    assert bool(torch.isfinite(want).all())
    none = lambda: None  # noqa: E731
    assert all(torch.equal(run(none), want) for _ in range(3))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run(none)
    for _ in range(3):
        graph.replay()
        assert torch.equal(captured, want)
    native.check_status()


def test_router_linear_and_top2(native):
    from b200moe import ops
    from b200moe.ops import functional as Fn
    T, D, E = 1000, 512, 8
    x = _rand(T, D).requires_grad_(True)
    w = _rand(E, D, scale=0.05).requires_grad_(True)
    logits = ops.linear(x, w)
    assert logits.dtype == torch.float32
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    lr = xr @ wr.t()
    assert _rel(logits, lr) < 1e-3
    weights, idx = ops.router_top2(logits)
    wref, iref = Fn.router_top2_ref(lr, 2)
    assert torch.equal(idx, iref) and _rel(weights, wref) < 1e-4
    dw = torch.randn(T, 2, device="cuda")
    weights.backward(dw)
    wref.backward(dw)
    assert _rel(x.grad, xr.grad) < 1e-2 and _rel(w.grad, wr.grad) < 1e-2


@pytest.mark.parametrize("T,N,K", [(1, 2, 8), (31, 5, 264), (33, 8, 520), (300, 9, 512), (2051, 16, 1032)])
def test_skinny_products(native, T, N, K):
    """Router-shaped products: token counts around the four-token and 32-token groups, outputs on both sides of eight,
    widths that leave lanes and column blocks partly empty.  fp32 sums of bf16 products: 1e-5; bf16 output: 2^-8."""
    torch.manual_seed(T)
    x, w = _rand(T, K), _rand(N, K)
    dy = torch.randn(T, N, device="cuda")
    assert _rel(native.gemm_nt(x, w).double(), x.double() @ w.double().t()) < 1e-5
    assert _rel(native.gemm_nn(dy, w).double(), dy.double() @ w.double()) < 4e-3
    base = torch.randn(N, K, device="cuda")
    got = native.gemm_tn(dy, x, out=base.clone(), accumulate=True)
    assert _rel(got.double() - base.double(), dy.double().t() @ x.double()) < 1e-5
    native.check_status()


@pytest.mark.parametrize("keep", [True, False])
def test_lm_head_without_a_known_factor_keeps_or_rebuilds_its_logits(native, keep, monkeypatch):
    """Both forms of the head against 64 bits, with a factor on the loss, twice through the same graph (nothing that
    the first backward pass read is changed by it), for a weight gradient and for an accumulator."""
    from b200moe import ops
    from b200moe.ops import loss as L
    if not keep:
        monkeypatch.setattr(L, "KEEP_BYTES", 0)
        monkeypatch.setattr(L, "CHUNK_TOKENS", 96)
    torch.manual_seed(3)
    T, D, V = 201, 128, 640
    hidden, weight = _rand(T, D).requires_grad_(True), _rand(V, D, scale=0.1).requires_grad_(True)
    targets = torch.randint(0, V, (T,), device="cuda")
    h64, w64 = (t.detach().double().requires_grad_(True) for t in (hidden, weight))
    (3 * torch.nn.functional.cross_entropy(h64 @ w64.t(), targets)).backward()
    loss = ops.lm_head_cross_entropy(hidden, weight, targets)
    for _ in range(2):
        hidden.grad = weight.grad = None
        (3 * loss).backward(retain_graph=True)
        # bf16 logits, dlogits and results: three roundings of 2^-9
        assert _rel(hidden.grad, h64.grad) < 8e-3 and _rel(weight.grad, w64.grad) < 8e-3
    weight.main_grad = torch.ones(V, D, device="cuda")
    hidden.grad = None
    (3 * ops.lm_head_cross_entropy(hidden, weight, targets)).backward()
    assert _rel(weight.main_grad - 1, w64.grad) < 8e-3 and _rel(hidden.grad, h64.grad) < 8e-3
    native.check_status()


@pytest.mark.parametrize("kept", [64, 128, 192])
def test_lm_head_keeps_the_chunks_that_fit_and_rebuilds_the_rest(native, kept, monkeypatch):
    """The same results as with all logits kept, up to the roundings of the rebuilt chunks (logits times the factor in
    bf16) and of a weight gradient that is added up in fp32: four of 2^-9."""
    from b200moe import ops
    from b200moe.ops import loss as L
    torch.manual_seed(3)
    T, D, V = 201, 128, 640
    targets, results = torch.randint(0, V, (T,), device="cuda"), []
    hidden, weight = _rand(T, D).requires_grad_(True), _rand(V, D, scale=0.1).requires_grad_(True)
    for limit in (L.KEEP_BYTES, 2 * V * (kept + 5)):
        monkeypatch.setattr(L, "KEEP_BYTES", limit)
        monkeypatch.setattr(L, "CHUNK_TOKENS", 64)
        assert L._kept_tokens(T, V) == (T if not results else kept)
        hidden.grad = weight.grad = None
        loss = ops.lm_head_cross_entropy(hidden, weight, targets)
        (3 * loss).backward()
        weight.main_grad = torch.ones(V, D, device="cuda")
        first = [loss.detach(), hidden.grad, weight.grad]
        hidden.grad = None
        (3 * ops.lm_head_cross_entropy(hidden, weight, targets)).backward()
        results.append(first + [hidden.grad, weight.main_grad - 1])
        del weight.main_grad
    for got, want in zip(*results):
        assert _rel(got, want) < 8e-3
    native.check_status()


@pytest.mark.parametrize("T,V", [(1, 8), (149, 8192), (300, 8200), (297, 16384), (150, 16392), (600, 32000), (149, 32768),
                                 (3, 32776)])
def test_cross_entropy_row_sizes(native, T, V):
    """Row sizes around those that select the kernel (2 and 4 vectors per thread, rows through shared memory, streaming
    beyond), more rows than CTAs, the first and the last entry as targets: against 64 bits.  Loss: fp32 sums; gradient:
    stored as bf16."""
    torch.manual_seed(V)
    logits = _rand(T, V, scale=2.0)
    targets = torch.randint(0, V, (T,), device="cuda")
    targets[0], targets[-1] = 0, V - 1
    l64 = logits.double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(l64, targets, reduction="sum") / T
    want.backward()
    loss = torch.zeros((), device="cuda")
    native.cross_entropy_scaled_(logits, targets, loss, 1.0 / T, 1.0 / T)
    assert abs(float(loss) - float(want)) < 1e-5 * abs(float(want))
    assert _rel(logits.double(), l64.grad) < 4e-3
    native.check_status()


@pytest.mark.parametrize("V", [2048, 32000, 33000])
def test_loss_does_not_depend_on_the_order_of_the_ctas(native, V):
    T = 1500
    logits, targets = _rand(T, V), torch.randint(0, V, (T,), device="cuda")
    want = torch.nn.functional.cross_entropy(logits.double(), targets)
    got = set()
    for _ in range(5):
        loss = torch.zeros((), dtype=torch.float64, device="cuda")
        native.cross_entropy_scaled_(logits.clone(), targets, loss, 1.0 / T, 1.0 / T)
        got.add(float(loss.float()))
    # rows: an fp32 sum of V exponentials, a logarithm and two additions, each good to a few 2^-24 of the row's loss
    assert len(got) == 1 and abs(got.pop() - float(want)) < 2e-6 * float(want)
    native.check_status()


def test_cross_entropy_and_lm_head(native):
    from b200moe import ops
    T, D, V = 512, 256, 32000
    h = _rand(2, T // 2, D).requires_grad_(True)
    w = _rand(V, D, scale=0.05).requires_grad_(True)
    t = torch.randint(0, V, (2, T // 2), device="cuda")
    loss = ops.lm_head_cross_entropy(h, w, t)
    hr, wr = h.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy((hr @ wr.t()).reshape(-1, V), t.reshape(-1))
    assert abs(float(loss) - float(ref)) < 2e-2
    (loss * 0.5).backward()
    (ref * 0.5).backward()
    assert _rel(h.grad, hr.grad) < 3e-2 and _rel(w.grad, wr.grad) < 3e-2


def test_lm_head_forms_its_gradients_in_the_forward_pass_when_the_loss_factor_is_known(native):
    """Three token chunks (one ragged); the weight gradient lands in ``main_grad`` with the announced factor."""
    from b200moe import ops
    T, D, V = 2 * 4096 + 640, 128, 4096
    h = _rand(T, D).requires_grad_(True)
    w = _rand(V, D, scale=0.05)
    w.main_grad = torch.zeros(V, D, device="cuda")
    t = torch.randint(0, V, (T,), device="cuda")
    hr, wr = h.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(hr @ wr.t(), t)
    (ref * 0.25).backward()
    for announced in (0.25, None):
        w.main_grad.zero_()
        h.grad = None
        loss = ops.lm_head_cross_entropy(h, w, t, grad_scale=announced)
        assert abs(float(loss) - float(ref)) < 2e-2
        (loss * 0.25).backward()
        assert _rel(h.grad, hr.grad) < 3e-2, announced
        assert _rel(w.main_grad, wr.grad) < 3e-2, announced


def test_many_tensors_per_optimizer_launch_and_zero_fill(native):
    """Sizes around the vector, the block and the 48-tensor table, mixed types and gradient factors: the update against
    the same arithmetic on the CPU, and the zero fill against a guard element on either side."""
    from b200moe.optim import AdamW
    torch.manual_seed(7)
    sizes = [1, 7, 8, 9, 8191, 8192, 8193, 16391] + [130] * 45
    gpu, cpu = [], []
    for i, n in enumerate(sizes):
        dtype = torch.bfloat16 if i % 3 == 0 else torch.float32
        p = torch.nn.Parameter(torch.randn(n, device="cuda").to(dtype))
        p.grad = torch.randn(n, device="cuda").to(dtype)
        q = torch.nn.Parameter(p.detach().cpu().clone())
        q.grad = p.grad.cpu().clone()
        if i % 5 == 0:
            p._grad_scale = q._grad_scale = 0.5
        gpu.append(p)
        cpu.append(q)
    a, b = AdamW(gpu, lr=1e-2), AdamW(cpu, lr=1e-2)
    before = native.launch_count()
    a.step()
    assert native.launch_count() - before == 4          # two types, two factors
    a.step()
    b.step()
    b.step()
    for p, q in zip(gpu, cpu):
        tol = 8e-3 if p.dtype == torch.bfloat16 else 1e-6
        assert _rel(p.detach().cpu(), q.detach()) < tol
        # the kernel forms 1 - beta2 in fp32: 0.999 is off by up to 2^-25, which is 3e-5 of 0.001
        assert _rel(a.state[p]["v"].cpu(), b.state[q]["v"]) < 4e-5
    spans = [torch.ones(n + 8, device="cuda", dtype=torch.bfloat16) for n in (1, 7, 8, 40000, 32760, 32768, 65537)] * 10
    spans = [t.clone() for t in spans]
    native.zero_many_([t[8:-1] if t.numel() > 9 else t[8:] for t in spans] + [spans[0][1:3]])
    for i, t in enumerate(spans):
        assert t[8:-1].abs().sum() == 0 and (t.numel() <= 9 or t[-1] == 1)
        assert t[:8].sum() == (6 if i == 0 else 8)
    native.check_status()


def test_zero_fill_of_whole_vectors_remainders_and_empty_buffers(native):
    """Buffers on 32-byte and on 16-byte boundaries, empty ones between and behind them, ends inside a thread's 32 bytes
    and around the 8 KiB of a CTA; guard bytes on either side stay."""
    sizes = [0, 1, 31, 32, 33, 0, 0, 8191, 8192, 8193, 100_000, 0]
    for shift in (32, 16):
        spans = [torch.full((n + 96,), 7, dtype=torch.uint8, device="cuda") for n in sizes]
        native.zero_many_([t[shift:shift + n] for t, n in zip(spans, sizes)])
        for t, n in zip(spans, sizes):
            assert not t[shift:shift + n].any()
            assert bool((t[:shift] == 7).all()) and bool((t[shift + n:] == 7).all())
    native.zero_many_([torch.empty(0, device="cuda")])
    native.check_status()


@pytest.mark.parametrize("total", [2047, 4097, 19_500_001])
def test_optimizer_blocks_of_both_sizes(native, total):
    """Blocks of 2048 elements, and of 8192 where they fill the machine (from 16 per SM): every element updated once, the
    remainder behind the last vector too.  fp32 arithmetic in another order: four roundings of 2^-24."""
    shapes = [total - total // 3, total // 3]
    p, g, m, v = ([torch.randn(n, device="cuda") for n in shapes] for _ in range(4))
    v = [t.abs() for t in v]
    want = []
    for a, b, c, d in zip(p, g, m, v):
        mean, square = 0.9 * c + 0.1 * b, 0.999 * d + 0.001 * b * b
        want.append((a * (1 - 1e-3 * 0.1) - 2e-3 * mean / (square.sqrt() + 1e-8), mean, square))
    native.adamw_many_([(*t, None) for t in zip(p, g, m, v)], 1e-3, 0.9, 0.999, 1e-8, 0.1, 2e-3)
    for got, exact in zip(zip(p, m, v), want):
        for a, b in zip(got, exact):
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-6)     # 1 - beta2 formed in fp32: 3e-5 of 0.001
    native.check_status()


def test_embedding_rope_adamw(native):
    from b200moe import ops
    from b200moe.ops import functional as Fn
    from b200moe.ops.attention import rope_qk_
    from b200moe.optim import AdamW
    table = _rand(1000, 128)
    table.main_grad = torch.zeros(1000, 128, device="cuda")
    table.requires_grad_(True)
    ids = torch.randint(0, 1000, (4, 33), device="cuda")
    out = ops.embedding(ids, table)
    assert torch.equal(out, table.detach()[ids])
    dy = _rand(4, 33, 128)
    out.backward(dy)
    want = torch.zeros(1000, 128, device="cuda").index_add_(0, ids.reshape(-1), dy.reshape(-1, 128).float())
    assert _rel(table.main_grad, want) < 1e-5
    # rope
    B, S, H, hd = 2, 64, 6, 128
    cos, sin = Fn.rope_tables(10000.0, hd, 128, device="cuda")
    qkv = _rand(B, S, H, hd).requires_grad_(True)
    rotated = rope_qk_((qkv * 1.0).view(B * S, H * hd), S, H, 4, hd, cos, sin).view(B, S, H, hd)
    ref_in = qkv.detach().float().requires_grad_(True)
    ref = torch.cat((Fn.apply_rope_ref(ref_in[:, :, :4].transpose(1, 2), cos[:S], sin[:S]).transpose(1, 2),
                     ref_in[:, :, 4:]), dim=2)
    assert _rel(rotated, ref) < 5e-3
    g = _rand(B, S, H, hd)
    rotated.backward(g)
    ref.backward(g.float())
    assert _rel(qkv.grad, ref_in.grad) < 5e-3
    # adamw: bf16 parameter with fp32 gradient accumulator and bf16 moments, and plain fp32
    for p_dt, g_dt, s_dt in [(torch.bfloat16, torch.float32, torch.bfloat16), (torch.float32, torch.float32, torch.float32),
                             (torch.bfloat16, torch.bfloat16, torch.float32)]:
        p = torch.nn.Parameter(torch.randn(4097, device="cuda").to(p_dt))
        cpu = torch.nn.Parameter(p.detach().cpu().clone())
        p.main_grad = torch.randn(4097, device="cuda").to(g_dt)
        cpu.main_grad = p.main_grad.cpu().clone()
        o1, o2 = AdamW([p], lr=1e-2, state_dtype=s_dt), AdamW([cpu], lr=1e-2, state_dtype=s_dt)
        for _ in range(3):
            o1.step()
            o2.step()
        assert _rel(p.detach().cpu(), cpu.detach()) < (1e-6 if p_dt == torch.float32 else 4e-3)


@pytest.mark.parametrize("T,E", [(257, 4), (1024, 8), (64, 8)])
def test_moe_plan_gather_combine(native, T, E):
    idx = torch.stack([torch.randperm(E, device="cuda")[:2] for _ in range(T)])
    if T == 64:
        idx[:] = torch.tensor([5, 2], device="cuda")          # everything on two experts
    from b200moe.ops.moe_fused import capacity_rows
    cap = capacity_rows(T * 2, E)
    slot_row, row_slot, offs, tile_expert, meta, counts = native.moe_plan(idx, E, cap)
    flat = idx.reshape(-1)
    assert torch.equal(counts.long(), torch.bincount(flat, minlength=E))
    ends = offs.tolist()
    assert int(meta[1]) == ends[-1] and int(meta[0]) == ends[-1] // 128 and int(meta[2]) == 0
    start = 0
    for e, end in enumerate(ends):
        slots_e = torch.nonzero(flat == e).flatten()
        assert torch.equal(slot_row[slots_e].long(), torch.arange(start, start + slots_e.numel(), device="cuda"))
        assert torch.equal(row_slot[start:start + slots_e.numel()].long(), slots_e)
        assert bool((row_slot[start + slots_e.numel():end] == -1).all())
        assert bool((tile_expert[start // 128:end // 128] == e).all())
        start = end
    x = _rand(T, 256)
    xp = native.moe_gather(x, row_slot, meta, cap)
    live = int(meta[1])
    want = torch.where(row_slot[:live, None] >= 0, x[(row_slot[:live].clamp_min(0) // 2).long()], torch.zeros_like(x[:1]))
    assert torch.equal(xp[:live], want)
    w = torch.rand(T, 2, device="cuda")
    out = native.moe_combine(xp, slot_row, w, T)
    assert _rel(out, x.float() * w.sum(1, keepdim=True)) < 5e-3


@pytest.mark.parametrize("T,E", [(1279, 8), (1280, 8), (5003, 16), (3000, 49), (2000, 1)])
def test_moe_plan_of_many_slots(native, T, E):
    """One CTA and a cluster of eight, runs of slots that end inside a warp, more experts than lanes."""
    from b200moe.ops.moe_fused import capacity_rows
    idx = torch.randint(0, E, (T, 2), device="cuda")
    slot_row, row_slot, offs, tile_expert, meta, counts = native.moe_plan(idx, E, capacity_rows(T * 2, E))
    flat = idx.reshape(-1)
    order = torch.argsort(flat, stable=True)
    want = torch.bincount(flat, minlength=E)
    ends = ((want + 255) // 256 * 256).cumsum(0)
    starts = ends - (want + 255) // 256 * 256
    rank = torch.arange(2 * T, device="cuda") - (want.cumsum(0) - want)[flat[order]]
    assert torch.equal(counts.long(), want) and torch.equal(offs.long(), ends)
    assert torch.equal(slot_row[order].long(), starts[flat[order]] + rank)
    live = int(ends[-1])
    rows = torch.full((live,), -1, device="cuda")
    rows[slot_row.long()] = torch.arange(2 * T, device="cuda")
    assert torch.equal(row_slot[:live].long(), rows) and meta[:3].tolist() == [live // 128, live, 0]
    assert torch.equal(tile_expert[:live // 128].long(), torch.repeat_interleave(torch.arange(E, device="cuda"), (ends - starts) // 128))


@pytest.mark.parametrize("offset", [0, 1, 4])
def test_embedding_gradient_on_and_off_a_16_byte_boundary(native, offset):
    T, V, D = 301, 40, 72
    ids, dy = torch.randint(0, V, (T,), device="cuda"), _rand(T, D)
    grad = torch.zeros(V * D + 8, device="cuda")
    native.embedding_bwd(ids, dy, grad[offset:offset + V * D].view(V, D))
    want = torch.zeros(V, D, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())
    scale = torch.zeros(V, D, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double().abs())
    got = grad[offset:offset + V * D].view(V, D)
    assert bool(((got.double() - want).abs() <= T * 2.0 ** -24 * scale).all())
    assert not grad[:offset].any() and not grad[offset + V * D:].any()


def test_combine_with_a_residual_rounds_like_the_sum_of_two_tensors(native):
    """A block's output decides the next router's choices, so the fused sum has to be the separate one bit for bit."""
    T, D = 1001, 264
    y, residual, w = _rand(2 * T, D), _rand(T, D), torch.rand(T, 2, device="cuda")
    slot_row = torch.randperm(2 * T, device="cuda").int()
    for weights in (w, None):
        fused = native.moe_combine(y, slot_row, weights, T, residual=residual)
        assert torch.equal(fused, residual + native.moe_combine(y, slot_row, weights, T))


@pytest.mark.parametrize("recompute", [False, True])
def test_moe_block_matches_torch_path(native, recompute):
    from b200moe import ops
    from b200moe.ops.moe import moe_ffn
    torch.manual_seed(1)
    T, D, Fd, E = 640, 256, 512, 4
    x = _rand(T, D)
    logits = torch.randn(T, E, device="cuda")
    w1, w3, w2 = _rand(E, Fd, D, scale=0.06), _rand(E, Fd, D, scale=0.06), _rand(E, D, Fd, scale=0.06)
    dout = _rand(T, D)
    results = []
    for use_native in (True, False):
        ops.set_native(use_native)
        try:
            xs = x.clone().requires_grad_(True)
            lg = logits.clone().requires_grad_(True)
            params = [p.clone().requires_grad_(True) for p in (w1, w2, w3)]
            weights, idx = ops.router_top2(lg)
            out = moe_ffn(xs, weights, idx, *params, recompute=recompute)
            out.backward(dout)
            results.append([out.detach(), xs.grad, lg.grad] + [p.grad for p in params])
        finally:
            ops.set_native(True)
    for got, want in zip(*results):
        assert _rel(got, want) < 2e-2
    native.check_status()


@pytest.mark.parametrize("keep_rows,recompute", [(None, False), (512, False), (None, True)])
def test_moe_block_with_fused_exchange_on_a_single_rank_group(native, tile_mode, keep_rows, recompute):
    """The gather+GEMM kernels, the return in the GEMM epilogue and the combine kernel with every pointer local
    (expert group of one rank), against the PyTorch statements of the block."""
    from b200moe import ops
    from b200moe.comm.ep import EPPull
    from b200moe.ops.moe import moe_ffn
    from b200moe.ops.moe_fused import moe_ffn_pull
    torch.manual_seed(3)
    T, D, Fd, E = 1000 if keep_rows is None else 1024, 256, 512, 4
    T = 1024
    x = _rand(T, D)
    logits = torch.randn(T, E, device="cuda")
    logits[:, 1] += 1.0
    w1, w3, w2 = _rand(E, Fd, D, scale=0.06), _rand(E, Fd, D, scale=0.06), _rand(E, D, Fd, scale=0.06)
    dout = _rand(T, D)
    epc = EPPull(None, native.status_word(), torch.device("cuda", torch.cuda.current_device()), T, D, Fd, E)
    if keep_rows is not None:
        epc.expected_rows = lambda key: keep_rows
    results = []
    for fused in (True, False, True):
        xs = x.clone().requires_grad_(True)
        lg = logits.clone().requires_grad_(True)
        params = [p.clone().requires_grad_(True) for p in (w1, w2, w3)]
        if fused:
            out, _, _ = moe_ffn_pull(xs, lambda staged: ops.router_top2(lg), *params, epc, recompute=recompute)
        else:
            ops.set_native(False)
            try:
                weights, idx = ops.router_top2(lg)
                out = moe_ffn(xs, weights, idx, *params)
            finally:
                ops.set_native(True)
        out.backward(dout)
        results.append([out.detach(), xs.grad, lg.grad] + [p.grad for p in params])
    for got, want, again in zip(*results):
        assert _rel(got, want) < 2e-2
        assert _rel(again, want) < 2e-2
    assert len(epc.free) == len(epc.pool) == 1
    native.check_status()


@pytest.mark.parametrize("T,E", [(1, 2), (33, 8), (257, 9), (130, 16)])
@pytest.mark.parametrize("aux", [False, True])
def test_routed_layer_as_one_op_against_its_separate_steps(native, T, E, aux):
    """Router, experts and the residual as one op against the separate router, top-2 and expert ops (a hook on the
    router sends the layer there): token counts around the four-token groups, experts on both sides of eight.  The two
    round the input gradient and the sum with the residual differently: three roundings of 2^-9."""
    from b200moe.models.layers import MoELayerMulti
    torch.manual_seed(T)
    D, F = 128, 256
    with torch.device("cuda"):
        layer = MoELayerMulti(D, F, num_expert_per_node=E)
    layer.router.compute_weight = layer.router.weight.detach().bfloat16().requires_grad_(True)
    router = layer.router.compute_weight
    x, residual, dy = _rand(T, D), _rand(T, D), _rand(T, D)
    results = []
    for separate in (False, True):
        handle = layer.router.register_forward_hook(lambda *_: None) if separate else None
        leaves = [t.clone().requires_grad_(True) for t in (x, residual)]
        for p in (*layer.experts.parameters(), router):
            p.grad = None
        out = layer._forward(leaves[0], aux, leaves[1])
        out, extra = out if aux else (out, None)
        torch.autograd.backward([out] + ([extra] if aux else []), [dy] + ([torch.full_like(extra, 0.5)] if aux else []))
        assert (type(out.grad_fn.next_functions[0][0]).__name__ == "_MoELayerBackward") or separate
        results.append([out.detach(), *([extra.detach()] if aux else []), leaves[0].grad, leaves[1].grad, router.grad,
                        *(p.grad for p in layer.experts.parameters())])
        if handle:
            handle.remove()
    for got, want in zip(*results):
        assert _rel(got, want) < 8e-3
    native.check_status()


def test_tiny_model_native_vs_torch_path(native):
    from b200moe import ops
    from b200moe.models import TransformerLMPipelined
    from b200moe.ops.functional import cross_entropy
    from b200moe.optim import AdamW
    from b200moe.parallel import FSDPWrapperPipelined, pipelined_train_overlap
    losses = []
    for use_native in (True, False):
        ops.set_native(use_native)
        try:
            torch.manual_seed(3)
            model = TransformerLMPipelined(2048, 256, 512, 2, 4, 0, 1, num_expert_per_node=4, d_ff=1024).cuda()
            wrapped = FSDPWrapperPipelined(model, None, None, compute_dtype=torch.bfloat16)
            opt = AdamW(wrapped.parameters(), lr=1e-3, weight_decay=0.01)
            ids = torch.randint(0, 2048, (4, 257), device="cuda")
            run = []
            for _ in range(4):
                run.append(float(pipelined_train_overlap(wrapped, opt, ids[:, :-1], ids[:, 1:], [4, 256, 512], 2, 0,
                                                         cross_entropy, dtype=torch.bfloat16, device=ids.device)))
            losses.append(run)
        finally:
            ops.set_native(True)
    assert losses[0][-1] < losses[0][0]
    assert losses[0] == pytest.approx(losses[1], abs=5e-2)
    native.check_status()
    assert native.launch_count() > 0


@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 128, 4, 1), (2, 512, 8, 2), (1, 1024, 4, 4)])
def test_attention_forward_backward(native, B, S, Hq, Hkv):
    from b200moe.ops import functional as Fn
    torch.manual_seed(2)
    hd, total = 128, Hq + 2 * Hkv
    qkv = _rand(B, S, total, hd)
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    out, lse, _, _ = native.attention_fwd(q, k, v)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = Fn.attention_ref(qf, kf, vf, None, None, causal=True)
    assert _rel(out, ref) < 1e-2
    scores = torch.einsum("bshd,bthd->bhst", qf, kf.repeat_interleave(Hq // Hkv, 2)) / math.sqrt(hd)
    scores = scores.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1), float("-inf"))
    assert _rel(lse, torch.logsumexp(scores, -1)) < 1e-3
    dout = _rand(B, S, Hq, hd)
    dq, dk, dv = native.attention_bwd(dout, q, k, v, out, lse)
    ref.backward(dout.float())
    assert _rel(dq, qf.grad) < 2e-2 and _rel(dk, kf.grad) < 2e-2 and _rel(dv, vf.grad) < 2e-2
    native.check_status()


def test_attention_at_the_training_shape_against_fp32_one_kv_group_at_a_time(native):
    """Sequence 8192 with 32 query and 8 key/value heads: the fp32 statement is evaluated per key/value head (four
    query heads, a 4 x 8192 x 8192 score block) so that it fits beside the kernels' tensors."""
    torch.manual_seed(4)
    B, S, Hq, Hkv, hd = 1, 8192, 32, 8, 128
    ratio, total = Hq // Hkv, Hq + 2 * Hkv
    qkv = _rand(B, S, total, hd)
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    dout = _rand(B, S, Hq, hd)
    out, lse, _, _ = native.attention_fwd(q, k, v)
    dq, dk, dv = native.attention_bwd(dout, q, k, v, out, lse)
    native.check_status()
    mask = torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1)
    for g in range(Hkv):
        heads = slice(g * ratio, (g + 1) * ratio)
        qf = q[0, :, heads].detach().float().transpose(0, 1).requires_grad_(True)       # [4, S, hd]
        kf = k[0, :, g].detach().float().requires_grad_(True)                           # [S, hd]
        vf = v[0, :, g].detach().float().requires_grad_(True)
        scores = (qf @ kf.t()) / math.sqrt(hd)
        scores = scores.masked_fill(mask, float("-inf"))
        ref = torch.softmax(scores, -1) @ vf                                             # [4, S, hd]
        ref.backward(dout[0, :, heads].float().transpose(0, 1))
        assert _rel(out[0, :, heads].transpose(0, 1), ref) < 1e-2, g
        assert _rel(lse[0, heads], torch.logsumexp(scores.detach(), -1)) < 1e-3, g
        assert _rel(dq[0, :, heads].transpose(0, 1), qf.grad) < 2e-2, g
        assert _rel(dk[0, :, g], kf.grad) < 2e-2 and _rel(dv[0, :, g], vf.grad) < 2e-2, g
        del scores, ref, qf, kf, vf


@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 256, 2, 2), (2, 512, 4, 1)])
def test_attention_non_causal(native, B, S, Hq, Hkv):
    """Every query sees every key (the form of the reference's own flash kernel): forward and backward."""
    from b200moe.ops import functional as Fn
    from b200moe.ops.attention import attention
    torch.manual_seed(4)
    hd = 128
    q, k, v = (_rand(B, S, h, hd).requires_grad_(True) for h in (Hq, Hkv, Hkv))
    out = attention(q, k, v, causal=False)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = Fn.attention_ref(qf, kf, vf, None, None, causal=False)
    assert _rel(out, ref) < 1e-2
    dout = _rand(B, S, Hq, hd)
    out.backward(dout)
    ref.backward(dout.float())
    assert _rel(q.grad, qf.grad) < 2e-2 and _rel(k.grad, kf.grad) < 2e-2 and _rel(v.grad, vf.grad) < 2e-2
    native.check_status()


@pytest.mark.parametrize("S", [1, 100, 127, 129, 257, 387])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_of_ragged_sequences(native, S, causal):
    """Sequences around the 128-row tile edges (one and two query tiles per CTA, a masked last key tile), with rotation
    where causal.  The second batch entry starts with non-finite rows: the first one's last tile must not read them.
    Bounds as for whole tiles: bf16 inputs, probabilities and outputs."""
    from b200moe.ops import functional as Fn, rope_attention
    from b200moe.ops.attention import attention
    torch.manual_seed(S)
    B, Hq, Hkv, hd = 2, 4, 2, 128
    cos, sin = Fn.rope_tables(10000.0, hd, 512, device="cuda")
    q, k, v = (_rand(B, S, h, hd) for h in (Hq, Hkv, Hkv))
    dout = _rand(B, S, Hq, hd)
    for t in (q, k, v, dout):
        t[1, 0] = float("inf")
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    before = native.launch_count()
    out = rope_attention(*leaves, cos, sin) if causal else attention(*leaves, causal=False)
    out.backward(dout)
    assert native.launch_count() >= before + 4
    exact = [t.detach()[:1].double().requires_grad_(True) for t in leaves]
    heads = [t.transpose(1, 2) for t in exact]
    if causal:
        def turn(x):
            a, b, c, s_ = x[..., 0::2], x[..., 1::2], cos[:S].double(), sin[:S].double()
            return torch.stack((a * c - b * s_, a * s_ + b * c), -1).flatten(-2)
        heads[0], heads[1] = turn(heads[0]), turn(heads[1])
    kh, vh = (t.repeat_interleave(Hq // Hkv, 1) for t in heads[1:])
    scores = heads[0] @ kh.mT / math.sqrt(hd)
    if causal:
        scores = scores.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1), float("-inf"))
    ref = (scores.softmax(-1) @ vh).transpose(1, 2)
    ref.backward(dout[:1].double())
    assert _rel(out[:1], ref) < 1e-2
    for got, want in zip(leaves, exact):
        # dq and dk vanish where a row sees one key only: what is left is the rounding of dP - rowsum(dO O)
        floor = 2e-2 * float(want.grad.norm()) + (1e-2 * math.sqrt(want.numel()) if S == 1 else 0.0)
        assert float((got.grad[:1].double() - want.grad).norm()) <= floor
    native.check_status()


@pytest.mark.parametrize("S", [1, 128, 129, 200, 256, 257, 387, 640])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attention_forward_does_not_depend_on_the_size_of_the_grid(native, S, causal, dtype):
    """One sequence on the kernel for grids of one wave, and the same sequence in a batch that takes the kernel with two
    query tiles per CTA: the same bits.  The next batch entry is not finite: a last tile must not read its rows."""
    torch.manual_seed(S)
    H = 2
    B = torch.cuda.get_device_properties(0).multi_processor_count // (H * ((S + 127) // 128)) + 2
    q, k, v = (torch.randn(B, S, H, 128, device="cuda").to(dtype) for _ in range(3))
    q[:, :, 0] *= 4                                   # row maxima that grow by more than the rescaling threshold
    for t in (q, k, v):
        t[1] = float("inf")
    alone, alone_lse, _, _ = native.attention_fwd(q[:1], k[:1], v[:1], causal=causal)
    batch, batch_lse, _, _ = native.attention_fwd(q, k, v, causal=causal)
    assert bool(torch.isfinite(alone).all()) and bool(torch.isfinite(alone_lse).all())
    assert torch.equal(batch[0], alone[0]) and torch.equal(batch_lse[0], alone_lse[0])
    native.check_status()


@pytest.mark.parametrize("S", [128, 384])
@pytest.mark.parametrize("causal", [True, False])
def test_flash_attention_in_fp16_keeps_fp16_precision(native, S, causal):
    """fp16 inputs are multiplied as fp16: against 64 bits the error is that of fp16 probabilities and outputs (2^-11
    each), which a pass through bf16 (2^-9 per input) cannot reach."""
    from b200moe.ops.attention import flash_attention_forward
    torch.manual_seed(S)
    q, k, v = (torch.randn(2, 3, S, 128, device="cuda").half() for _ in range(3))
    scores = q.double() @ k.double().mT / math.sqrt(128)
    if causal:
        scores = scores.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1), float("-inf"))
    got = flash_attention_forward(q, k, v, causal=causal)
    assert got.dtype == torch.float16
    want = scores.softmax(-1) @ v.double()
    assert float((got.double() - want).norm() / want.norm()) < 1e-3
    native.check_status()


@pytest.mark.parametrize("B,S,Hq,Hkv,causal", [(1, 640, 4, 4, False), (1, 640, 2, 2, True), (2, 1024, 4, 1, True),
                                               (1, 1100, 8, 2, True), (1, 1025, 2, 2, False), (1, 896, 2, 2, True),
                                               (1, 4224, 1, 1, True), (1, 1152, 4, 4, False), (1, 1152, 16, 4, True)])
def test_attention_backward_shared_by_a_cluster(native, B, S, Hq, Hkv, causal):
    """Tiles whose steps two or four CTAs share: uneven parts, CTAs without a step, a ragged last tile."""
    q, k, v, dy = (_rand(B, S, h, 128) for h in (Hq, Hkv, Hkv, Hq))
    out, lse, _, _ = native.attention_fwd(q, k, v, causal=causal)
    got = native.attention_bwd(dy, q, k, v, out, lse, causal=causal)
    again = native.attention_bwd(dy, q, k, v, out, lse, causal=causal)
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    qh, kh, vh = (t.transpose(1, 2) for t in leaves)
    kh, vh = (t.repeat_interleave(Hq // Hkv, 1) for t in (kh, vh))
    scores = qh @ kh.mT * 128 ** -0.5
    if causal:
        scores = scores.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    want = torch.autograd.grad((scores.softmax(-1) @ vh).transpose(1, 2), leaves, dy.double())
    for a, b, c in zip(got, again, want):
        assert torch.equal(a, b) and _rel(a, c) < 1e-2
        # P and dS are rounded to bf16 (2^-9 each), the row statistic comes from a rounded output
        rows = (a.double() - c).norm(dim=-1) / (c.norm(dim=-1) + c.norm(dim=-1).mean())
        assert float(rows.max()) < 3e-2
    native.check_status()


def test_flash_attention_forward_entry(native):
    """``[B, H, S, 128]`` forward-only entry point, fp16 in and out, against an fp32 softmax(QK^T)V."""
    from b200moe.ops.attention import flash_attention_forward
    torch.manual_seed(5)
    B, H, S, hd = 2, 3, 384, 128
    q, k, v = (torch.randn(B, H, S, hd, device="cuda").half() for _ in range(3))
    before = native.launch_count()
    out = flash_attention_forward(q, k, v)
    assert native.launch_count() > before and out.dtype == torch.float16 and out.shape == (B, H, S, hd)
    ref = torch.softmax(q.float() @ k.float().transpose(-1, -2) / math.sqrt(hd), -1) @ v.float()
    assert _rel(out, ref) < 2e-2
    causal = flash_attention_forward(q, k, v, causal=True)
    mask = torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1)
    ref = torch.softmax((q.float() @ k.float().transpose(-1, -2) / math.sqrt(hd)).masked_fill(mask, float("-inf")), -1) @ v.float()
    assert _rel(causal, ref) < 2e-2
    native.check_status()


@pytest.mark.parametrize("causal", [False, True])
def test_reference_named_attention_functions_run_the_flash_kernels(native, causal):
    """``FlashAttentionTritonFunc.apply(q, k, v, is_causal)`` and the ``attention_forward[grid](...)`` launch of the
    reference's module, on bf16 ``[B, S, 128]`` tensors: forward and backward against an fp32 formula."""
    from implementation.kernels.attention import FlashAttentionTritonFunc, attention_forward
    torch.manual_seed(9)
    B, S, hd = 3, 256, 128
    q, k, v = (_rand(B, S, hd).requires_grad_(True) for _ in range(3))
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    scores = qf @ kf.transpose(-1, -2) / math.sqrt(hd)
    if causal:
        scores = scores.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1), float("-inf"))
    ref = torch.softmax(scores, -1) @ vf
    before = native.launch_count()
    out = FlashAttentionTritonFunc.apply(q, k, v, causal)
    assert native.launch_count() > before and out.shape == (B, S, hd) and out.dtype == torch.bfloat16
    assert _rel(out, ref) < 2e-2
    dout = _rand(B, S, hd)
    before = native.launch_count()
    out.backward(dout)
    assert native.launch_count() > before
    ref.backward(dout.float())
    assert _rel(q.grad, qf.grad) < 3e-2 and _rel(k.grad, kf.grad) < 3e-2 and _rel(v.grad, vf.grad) < 3e-2
    filled, lse = torch.empty(B, S, hd, device="cuda", dtype=torch.bfloat16), torch.empty(B, S, device="cuda")
    attention_forward[(S // 16, B)](q.detach(), k.detach(), v.detach(), filled, lse, *([0] * 14), S, S,
                                    1 / math.sqrt(hd), hd, 16, 16, causal)
    assert _rel(filled, ref) < 2e-2 and _rel(lse, torch.logsumexp(scores.detach(), -1)) < 1e-3
    native.check_status()


def test_fused_qkv_attention_with_rope(native):
    from b200moe.ops import functional as Fn
    from b200moe.ops.attention import fused_qkv_attention
    B, S, Hq, Hkv, hd = 2, 256, 8, 2, 128
    total = Hq + 2 * Hkv
    cos, sin = Fn.rope_tables(10000.0, hd, S, device="cuda")
    base = _rand(B * S, total * hd).requires_grad_(True)
    out = fused_qkv_attention(base * 1.0, B, S, Hq, Hkv, hd, cos, sin)
    ref_in = base.detach().float().requires_grad_(True)
    view = ref_in.view(B, S, total, hd)
    ref = Fn.attention_ref(view[:, :, :Hq], view[:, :, Hq:Hq + Hkv], view[:, :, Hq + Hkv:], cos, sin, causal=True)
    assert _rel(out, ref) < 1e-2
    g = _rand(B, S, Hq, hd)
    out.backward(g)
    ref.backward(g.float())
    assert _rel(base.grad, ref_in.grad) < 2e-2
    native.check_status()


@pytest.mark.parametrize("S", [100, 129, 387])
@pytest.mark.parametrize("in_epilogue", [False, True])
def test_fused_projection_and_attention_of_ragged_sequences(native, S, in_epilogue, monkeypatch):
    """The rotation by position = row mod S (in place, or in the projection's epilogue), and attention on strided slices
    of one buffer, where the rows behind a sequence belong to the next one: every row of the output and of the one
    gradient buffer (filled with NaN first) against 64 bits.  Bound per row: bf16 inputs, probabilities, products and
    results, as for whole tiles, against the mean row."""
    from b200moe import ops
    from b200moe.ops import functional as Fn
    from b200moe.ops.attention import fused_qkv_attention
    torch.manual_seed(S)
    B, Hq, Hkv, hd, D = 3, 4, 1, 128, 256
    total = Hq + 2 * Hkv
    cos, sin = Fn.rope_tables(10000.0, hd, 512, device="cuda")
    x, w, g = _rand(B * S, D), _rand(total * hd, D, scale=D ** -0.5), _rand(B, S, Hq, hd)
    if in_epilogue:
        qkv = ops.linear_rope(x, w, cos, sin, (Hq + Hkv) * hd, S)
    else:
        qkv = native.gemm_nt(x, w)
    leaf = qkv.detach().requires_grad_(True)
    plain = native.gemm_nt(x, w).double().requires_grad_(True)
    heads = [t.transpose(1, 2) for t in plain.view(B, S, total, hd).split((Hq, Hkv, Hkv), dim=2)]

    def turn(t):
        a, b, c, s_ = t[..., 0::2], t[..., 1::2], cos[:S].double(), sin[:S].double()
        return torch.stack((a * c - b * s_, a * s_ + b * c), -1).flatten(-2)

    scores = turn(heads[0]) @ turn(heads[1]).repeat_interleave(Hq // Hkv, 1).mT / math.sqrt(hd)
    hidden = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
    ref = (scores.masked_fill(hidden, -math.inf).softmax(-1) @ heads[2].repeat_interleave(Hq // Hkv, 1)).transpose(1, 2)
    ref.backward(g.double())
    empty_like = torch.empty_like
    monkeypatch.setattr(torch, "empty_like", lambda t, **kw: empty_like(t, **kw).fill_(float("nan")))
    out = fused_qkv_attention(leaf * 1.0, B, S, Hq, Hkv, hd, cos, sin, pre_rotated=in_epilogue)
    out.backward(g)
    for got, want in ((out.reshape(B * S, -1), ref.reshape(B * S, -1)), (leaf.grad, plain.grad)):
        rows = want.norm(dim=1)
        assert bool(torch.isfinite(got).all())
        assert float(((got.double() - want).norm(dim=1) / (rows + rows.mean())).max()) < 2e-2
    native.check_status()


@pytest.mark.parametrize("causal", [True, False])
def test_second_derivatives_of_ragged_attention(native, causal):
    """``create_graph=True`` at a length that is no multiple of 128: gradients of the gradients through the formula, where
    the library has a differentiable backward pass for it.  Bounds as for the gradients."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from b200moe.ops.attention import attention
    torch.manual_seed(9)
    B, S, H, hd = 1, 100, 2, 128
    leaves = [_rand(B, S, H, hd).requires_grad_(True) for _ in range(3)]
    dout, mix = _rand(B, S, H, hd), [_rand(B, S, H, hd) for _ in range(3)]

    def second(inputs, forward, weight):
        first = torch.autograd.grad(forward(*inputs), inputs, weight, create_graph=True)
        return torch.autograd.grad(sum((f * m.to(f.dtype)).sum() for f, m in zip(first, mix)), inputs)

    def formula(q, k, v):
        q, k, v = (t.transpose(1, 2) for t in (q, k, v))
        scores = q @ k.mT / math.sqrt(hd)
        if causal:
            scores = scores.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), -math.inf)
        return (scores.softmax(-1) @ v).transpose(1, 2)

    with sdpa_kernel(SDPBackend.MATH):
        got = second(leaves, lambda *t: attention(*t, causal=causal), dout)
    want = second([t.detach().double().requires_grad_(True) for t in leaves], formula, dout.double())
    for a, b in zip(got, want):
        assert _rel(a, b) < 2e-2
    native.check_status()


@pytest.mark.parametrize("tile", [0, 3], ids=["tiles_auto", "tiles_cta_pair"])
def test_projection_with_rope_in_the_gemm_epilogue_then_attention(native, tile):
    """q/k/v projection whose epilogue rotates q and k, attention on the rotated tensors, and a backward pass whose
    attention kernels hand back gradients of the unrotated projection: against the fp32 statements end to end."""
    from b200moe import ops
    from b200moe.ops import functional as Fn
    from b200moe.ops.attention import fused_qkv_attention
    native.set_gemm_tile_mode(tile)
    try:
        B, S, Hq, Hkv, hd, D = 2, 256, 8, 2, 128, 512
        total = Hq + 2 * Hkv
        cos, sin = Fn.rope_tables(10000.0, hd, 2 * S, device="cuda")       # a table longer than the sequence
        x = _rand(B * S, D).requires_grad_(True)
        w = _rand(total * hd, D, scale=0.05).requires_grad_(True)
        qkv = ops.linear_rope(x, w, cos, sin, (Hq + Hkv) * hd, S)
        xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
        plain = (xr @ wr.t()).view(B, S, total, hd)
        rotated = torch.cat([Fn.apply_rope_ref(plain[:, :, :Hq + Hkv].transpose(1, 2), cos[:S], sin[:S]).transpose(1, 2),
                             plain[:, :, Hq + Hkv:]], dim=2)
        assert _rel(qkv.view(B, S, total, hd), rotated) < 1e-2
        out = fused_qkv_attention(qkv, B, S, Hq, Hkv, hd, cos, sin, pre_rotated=True)
        ref = Fn.attention_ref(plain[:, :, :Hq], plain[:, :, Hq:Hq + Hkv], plain[:, :, Hq + Hkv:], cos[:S], sin[:S],
                               causal=True)
        assert _rel(out, ref) < 1.5e-2
        g = _rand(B, S, Hq, hd)
        out.backward(g)
        ref.backward(g.float())
        assert _rel(x.grad, xr.grad) < 3e-2 and _rel(w.grad, wr.grad) < 3e-2
        native.check_status()
    finally:
        native.set_gemm_tile_mode(0)


@pytest.mark.parametrize("S", [100, 129])
@pytest.mark.parametrize("fused", [True, False])
def test_attention_layer_of_ragged_sequences_rounds_like_the_library(native, S, fused):
    """Bit for bit the projection, the rotation and the library's attention one by one, with and without a fused
    projection weight: routers behind the layer turn another rounding into other choices."""
    from b200moe import ops
    from b200moe.models.layers import MultiHeadLayerLL, ROPELayer
    from b200moe.ops.attention import library_attention, rope_qk_
    torch.manual_seed(S)
    B, D, Hq, Hkv, hd = 2, 512, 4, 1, 128
    with torch.device("cuda"):
        layer = MultiHeadLayerLL(D, Hq, RoPE=ROPELayer(10000, hd, 256))
    for p in (layer.q_proj, layer.k_proj, layer.v_proj, layer.output_proj):
        p.compute_weight = p.weight.detach().bfloat16()
    q, k, v, out = (p.compute_weight for p in (layer.q_proj, layer.k_proj, layer.v_proj, layer.output_proj))
    x, cos, sin = _rand(B, S, D), layer.RoPE.cos, layer.RoPE.sin
    if fused:
        layer.qkv_weight = torch.cat((q, k, v))
        qkv = rope_qk_(ops.linear(x.view(B * S, D), layer.qkv_weight), S, Hq + 2 * Hkv, Hq + Hkv, hd, cos, sin)
        heads = qkv.view(B, S, Hq + 2 * Hkv, hd).split((Hq, Hkv, Hkv), dim=2)
        attended = library_attention(*heads, None, None)
    else:
        heads = [ops.linear(x, w).view(B, S, -1, hd) for w in (q, k, v)]
        attended = library_attention(*heads, cos, sin)
    assert torch.equal(layer(x), ops.linear(attended.reshape(B, S, D), out))
    native.check_status()


@pytest.mark.parametrize("M,K,world,segments", [(1000, 512, 2, [1536]), (300, 256, 2, [1984]),
                                                (2048, 1024, 4, [2048]), (700, 512, 2, [1024, 256, 256]),
                                                (513, 256, 4, [1024, 512, 512, 96 * 4])])
def test_allgather_gemm_emulated_ranks(native, M, K, world, segments):
    """The all-gather + GEMM kernel of every rank of a group, run one after the other on this GPU: each "rank" has
    its own full-size copy of W in which only its own rows are valid (the rest is NaN), the "peers" are the other
    copies, and the peers' ready signals are written by the host so that no launch waits for another one.
    ``segments``: stacked parts of W sharded one by one (a fused q/k/v projection has three)."""
    import ctypes
    torch.manual_seed(11)
    N = sum(segments)
    owner = torch.empty(N, dtype=torch.long)
    begin = 0
    for rows in segments:
        owner[begin:begin + rows] = torch.arange(rows) // (rows // world)
        begin += rows
    owner = owner.cuda()
    x = _rand(M, K)

    def fresh():
        full = _rand(N, K)
        parts = []
        for r in range(world):
            c = torch.full((N, K), float("nan"), dtype=torch.bfloat16, device="cuda")
            c[owner == r] = full[owner == r]
            parts.append(c)
        return full, parts

    W, filled = fresh()
    copies = [c.clone() for c in filled]
    table = ctypes.c_ulonglong * 8
    w_ptrs = table(*([c.data_ptr() for c in copies] + [0] * (8 - world)))
    pads = [torch.zeros(32 * 8, dtype=torch.int32, device="cuda") for _ in range(world)]
    sig_ptrs = table(*([s.data_ptr() for s in pads] + [0] * (8 - world)))
    slot = 14
    flags = [torch.zeros((N + 255) // 256, dtype=torch.int32, device="cuda") for _ in range(world)]
    for epoch in (1, 2):
        if epoch == 2:      # a second step: rows change, every copy is stale again outside its own rows
            W, filled = fresh()
        ref = x.float() @ W.float().t()
        for r in range(world):
            # what the ranks hold when rank r runs: their own rows only (nobody else has gathered yet)
            for q in range(world):
                copies[q].copy_(filled[q])
            pads[r].view(32, 8)[slot].fill_(epoch)      # "every peer has announced its rows"
            y = native.ag_gemm_nt(x, w_ptrs, N, segments, world, r, sig_ptrs, slot, epoch, flags[r], epoch)
            assert y is not None, "cooperative launch unavailable"
            native.check_status()
            assert _rel(y, ref) < 1e-2
            assert torch.equal(copies[r], W), "gathered weight differs from the sharded original"


def test_device_timestamp_and_step_timer(native):
    """``globaltimer`` stamps bracket the same span as CUDA events; NVTX wrapping of launches does not change results."""
    from b200moe.utils.profiling import DeviceStepTimer
    a, b = _rand(4096, 4096), _rand(4096, 4096)
    native.gemm_nt(a, b)
    torch.cuda.synchronize()
    by_event, by_clock = DeviceStepTimer("cuda"), DeviceStepTimer("cuda", clock="globaltimer")
    by_event.start()
    by_clock.start()
    for _ in range(20):
        native.gemm_nt(a, b)
    t_clock = by_clock.stop_ms()
    t_event = by_event.stop_ms()
    assert t_clock > 0 and abs(t_clock - t_event) < 0.25 * t_event + 0.05, (t_clock, t_event)
    native.set_nvtx(True)
    try:
        with_ranges = native.gemm_nt(a, b)
    finally:
        native.set_nvtx(False)
    assert torch.equal(with_ranges, native.gemm_nt(a, b))
    native.check_status()

