"""tcgen05 GEMM against an fp32 PyTorch reference: all operand layouts, ragged shapes, epilogues."""
import pytest
import torch

from atorch_b200 import _lib
from atorch_b200.ops import gemm, gemm_reference, linear

pytestmark = pytest.mark.gpu


def _mk(rows, cols, dev="cuda"):
    return (torch.randn(rows, cols, device=dev, dtype=torch.float32) * 0.5).to(torch.bfloat16)


def _check(out, ref, K):
    torch.cuda.synchronize()
    _lib.check_status(out.device)
    err = (out.float() - ref.float()).abs().max().item()
    scale = ref.float().abs().max().item() + 1e-6
    assert err / scale < 2e-2, f"max err {err} vs scale {scale}"


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 512, 256), (384, 264, 136), (1000, 1032, 520),
                                   (4096, 4096, 1024), (128, 4096, 4096), (72, 96, 40)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N + K)
    a = _mk(K, M) if a_mn else _mk(M, K)
    b = _mk(K, N) if b_mn else _mk(N, K)
    ref = gemm_reference(a, b, a_mn, b_mn, out_dtype=torch.float32)
    for tile_n in (128, 256):
        out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, tile_n=tile_n, kernel="1cta")
        _check(out, ref, K)
    for tile_n in (0, 128, 256):
        out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, kernel="2cta", tile_n=tile_n)
        _check(out, ref, K)


def test_gemm_fp32_out_accumulate_alpha_bias():
    torch.manual_seed(1)
    M, N, K = 512, 768, 384
    a, b = _mk(M, K), _mk(N, K)
    bias = _mk(1, N)[0]
    c0 = torch.randn(M, N, device="cuda")
    out = c0.clone()
    gemm(a, b, out=out, accumulate=True, alpha=0.5, bias=bias)
    ref = c0 + 0.5 * (a.float() @ b.float().t()) + bias.float()
    _check(out, ref, K)
    c1 = _mk(M, N)
    out = c1.clone()
    gemm(a, b, out=out, accumulate=True)
    _check(out, c1.float() + a.float() @ b.float().t(), K)


def test_gemm_strided_operands():
    torch.manual_seed(2)
    big = _mk(512, 1024)
    a = big[:, 256:768]  # pitch 1024, K = 512
    b = _mk(256, 512)
    out = gemm(a, b)
    _check(out, a.float() @ b.float().t(), 512)


def test_gemm_many_tiles_persistent():
    # more tiles than SMs: exercises accumulator double buffering and ring wrap-around
    torch.manual_seed(3)
    M, N, K = 4096, 11008, 512
    a, b = _mk(M, K), _mk(N, K)
    out = gemm(a, b)
    idx = torch.randint(0, M, (64,), device="cuda")
    ref = a[idx].float() @ b.float().t()
    _check(out[idx], ref, K)
    out2 = gemm(a, b, max_ctas=7)
    assert torch.equal(out, out2)
    out3 = gemm(a, b, kernel="1cta")
    _check(out3[idx], ref, K)
    c0 = torch.randn(M, N, device="cuda")
    o4 = c0.clone()
    gemm(a, b, out=o4, accumulate=True, alpha=0.5, kernel="2cta")
    _check(o4[idx], c0[idx] + 0.5 * ref, K)


def test_residual_epilogue():
    torch.manual_seed(6)
    M, N, K = 512, 4096, 256
    a, b, r = _mk(M, K), _mk(N, K), _mk(M, N)
    for kern in ("1cta", "2cta"):
        out = gemm(a, b, residual=r, kernel=kern)
        _check(out, r.float() + a.float() @ b.float().t(), K)


def test_linear_autograd_matches_torch():
    torch.manual_seed(4)
    x = _mk(96, 256).requires_grad_()
    w = _mk(512, 256).requires_grad_()
    res = _mk(96, 512).requires_grad_()
    y = linear(x, w, residual=res)
    dy = _mk(96, 512)
    y.backward(dy)
    xr, wr, rr = (t.detach().float().requires_grad_() for t in (x, w, res))
    yr = rr + xr @ wr.t()
    yr.backward(dy.float())
    _check(y, yr, 256)
    _check(x.grad, xr.grad, 512)
    _check(w.grad, wr.grad, 96)
    assert torch.equal(res.grad, dy)


def test_linear_main_grad_accumulation():
    torch.manual_seed(5)
    x = _mk(128, 256).requires_grad_()
    w = _mk(384, 256).requires_grad_()
    w.main_grad = torch.zeros(384, 256, device="cuda", dtype=torch.float32)
    dy = _mk(128, 384)
    for _ in range(2):
        linear(x, w).backward(dy)
    assert w.grad is None
    ref = 2 * (dy.float().t() @ x.detach().float())
    _check(w.main_grad, ref, 128)


def test_grouped_gemm_with_device_counts():
    """ops.gemm(groups=...): slot groups filled up to device-resident counts (zero beyond), empty tiles
    skipped and written as zeros, one stacked B operand per expert, k-block skipping in the wgrad form."""
    from atorch_b200 import ops

    torch.manual_seed(4)
    E, W, cap, K, N = 2, 3, 512, 256, 384
    G = E * W
    counts = torch.tensor([512, 0, 130, 256, 257, 1], dtype=torch.int32, device="cuda")
    x = torch.randn(G * cap, K, device="cuda", dtype=torch.bfloat16)
    rows = torch.arange(G * cap, device="cuda")
    valid = (rows % cap) < counts[rows // cap]
    x[~valid] = 0
    w = (0.1 * torch.randn(E, N, K, device="cuda")).bfloat16()
    out = torch.full((G * cap, N), 7.0, device="cuda", dtype=torch.bfloat16)      # stale contents everywhere
    ops.gemm(x, w.reshape(E * N, K), out=out, groups={"counts": counts, "m_rows": cap, "n_b": E, "bm_rows": W * cap})
    ref = torch.cat([x[e * W * cap:(e + 1) * W * cap].float() @ w[e].float().t() for e in range(E)])
    assert torch.allclose(out.float(), ref, rtol=2e-2, atol=2e-2)
    assert (out[~valid] == 0).all()
    # dgrad form: B read MN-major, stacked along its row (k) axis
    dy = torch.randn(G * cap, N, device="cuda", dtype=torch.bfloat16)
    dy[~valid] = 0
    dx = ops.gemm(dy, w.reshape(E * N, K), b_mn=True, groups={"counts": counts, "m_rows": cap, "n_b": E,
                                                                "bm_rows": W * cap})
    ref = torch.cat([dy[e * W * cap:(e + 1) * W * cap].float() @ w[e].float() for e in range(E)])
    assert torch.allclose(dx.float(), ref, rtol=2e-2, atol=3e-2)
    # wgrad form: the reduction runs over the slots, empty k-blocks are skipped
    for e in range(E):
        sl = slice(e * W * cap, (e + 1) * W * cap)
        dw = ops.gemm(dy[sl], x[sl], a_mn=True, b_mn=True, groups={"counts": counts[e * W:(e + 1) * W], "k_rows": cap})
        ref = dy[sl].float().t() @ x[sl].float()
        assert torch.allclose(dw.float(), ref, rtol=2e-2, atol=2e-1), (dw.float() - ref).abs().max()
    # all groups empty: zeros, not stale data
    zc = torch.zeros(W, dtype=torch.int32, device="cuda")
    dw = torch.full((N, K), 3.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm(dy[:W * cap], x[:W * cap], a_mn=True, b_mn=True, out=dw, groups={"counts": zc, "k_rows": cap})
    assert (dw == 0).all()


@pytest.mark.parametrize("T,H,F", [(512, 1024, 1408), (1000, 512, 2752), (4096, 4096, 11008)])
def test_linear_swiglu_epilogue_matches_separate_kernels(T, H, F):
    """SwiGLU in the GEMM epilogue: the activation and the kept gate|up tensor are bit-identical to the GEMM
    followed by the SwiGLU kernel, with and without gradients; gradients agree with the two-op form."""
    from atorch_b200 import ops

    torch.manual_seed(T + F)
    x = _mk(T, H)
    w = (_mk(2 * F, H) * 0.1).to(torch.bfloat16)
    with torch.no_grad():
        ref = ops.swiglu(ops.linear(x, w))
        out = ops.linear_swiglu(x, w)
    torch.cuda.synchronize()
    _lib.check_status(x.device)
    assert torch.equal(out, ref)
    xa, wa = x.clone().requires_grad_(), w.clone().requires_grad_()
    xb, wb = x.clone().requires_grad_(), w.clone().requires_grad_()
    ya = ops.linear_swiglu(xa, wa)
    yb = ops.swiglu(ops.linear(xb, wb))
    assert type(ya.grad_fn).__name__ == "_LinearSwiGLUBackward" and torch.equal(ya, yb)
    dy = _mk(T, F)
    ya.backward(dy)
    yb.backward(dy)
    torch.cuda.synchronize()
    _lib.check_status(x.device)
    assert torch.equal(xa.grad, xb.grad) and torch.equal(wa.grad, wb.grad)
    # against fp32 math
    g = x.float() @ w.float().t()
    full = torch.nn.functional.silu(g[:, :F]) * g[:, F:]
    _check(out, full, H)


def test_dynamic_tile_schedule_matches_static():
    """Tiles handed out by the atomic counter give bit-identical results to the fixed-stride schedule, launch after
    launch (the counters are left at zero), on two streams at once, and while another kernel shares the SMs."""
    L = _lib.lib()
    torch.manual_seed(11)
    side = torch.cuda.Stream()
    try:
        for M, N, K, a_mn, b_mn in [(4096, 4096, 1024, False, False), (4096, 11008, 512, False, True),
                                    (2048 + 72, 4096 + 8, 1024 + 40, True, True), (8192, 8192, 256, False, False)]:
            a = _mk(K, M) if a_mn else _mk(M, K)
            b = _mk(K, N) if b_mn else _mk(N, K)
            L.atb_gemm_set_dynamic(0)
            ref = gemm(a, b, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
            L.atb_gemm_set_dynamic(1)
            outs = [gemm(a, b, a_mn=a_mn, b_mn=b_mn, kernel="2cta") for _ in range(3)]
            filler = torch.empty(64 << 20, device="cuda")
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):                       # a second stream has counters of its own
                for _ in range(4):
                    filler.normal_()
                other = gemm(a, b, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
            busy = gemm(a, b, a_mn=a_mn, b_mn=b_mn, kernel="2cta")
            torch.cuda.synchronize()
            _lib.check_status(ref.device)
            for o in outs + [other, busy]:
                assert torch.equal(o, ref)
    finally:
        L.atb_gemm_set_dynamic(1)


@pytest.mark.parametrize("M,N,K", [(1, 64, 72), (129, 264, 136), (255, 256, 64), (257, 512, 200), (777, 1032, 520)])
def test_gemm_odd_token_counts(M, N, K):
    """Token counts that are no multiple of 8: rows of A in forward and dgrad, the reduction dim in wgrad."""
    torch.manual_seed(M)
    x, w, dy = _mk(M, K), _mk(N, K), _mk(M, N)
    bias, res = _mk(1, N)[0], _mk(M, N)
    _check(gemm(x, w, bias=bias, residual=res), x.float() @ w.float().t() + bias.float() + res.float(), K)
    _check(gemm(dy, w, b_mn=True), dy.float() @ w.float(), N)
    _check(gemm(dy, x, a_mn=True, b_mn=True), dy.float().t() @ x.float(), M)
    c0 = torch.randn(N, K, device="cuda")
    out = c0.clone()
    gemm(dy, x, a_mn=True, b_mn=True, out=out, accumulate=True)
    _check(out, c0 + dy.float().t() @ x.float(), M)


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("sizes", [(0, 1, 255, 0), (257, 0, 64, 129, 3), (512, 513), (0, 0, 40)])
def test_grouped_gemm_ragged_groups(sizes, trans_b):
    """Groups of any length in one launch, against one fp32 product per group; rows past a group's end belong to the
    next one and must not be touched by it."""
    from atorch_b200.ops.moe import grouped_gemm

    torch.manual_seed(sum(sizes))
    G, K, N = len(sizes), 192, 328
    x = _mk(sum(sizes), K).requires_grad_(True)
    w = (torch.randn(G, N, K, device="cuda") if trans_b else torch.randn(G, K, N, device="cuda")).bfloat16()
    w.requires_grad_(True)
    dy = _mk(sum(sizes), N)
    y = grouped_gemm(x, w, sizes, trans_b)
    y.backward(dy)
    r = 0
    for g, n in enumerate(sizes):
        xs, ds, wg = x.detach()[r: r + n].float(), dy[r: r + n].float(), w.detach()[g].float()
        wk = wg.t() if trans_b else wg                              # [K, N]
        if n:
            _check(y.detach()[r: r + n], xs @ wk, K)
            _check(x.grad[r: r + n], ds @ wk.t(), N)
        dw = xs.t() @ ds
        _check(w.grad[g], dw.t() if trans_b else dw, max(n, 1))
        r += n


@pytest.mark.parametrize("T,H,E,k", [(1, 8, 4, 1), (37, 264, 4, 2), (513, 4096, 8, 2), (64, 2048, 8, 3)])
@pytest.mark.parametrize("probs", [torch.bfloat16, torch.float32, None])
def test_permute_unpermute_row_kernels(T, H, E, k, probs):
    """Row movement of a routed layer and its gradients against the tensor operations in fp32 (one bf16 rounding each)."""
    from atorch_b200.ops import moe as M

    torch.manual_seed(T)
    x, dout = _mk(T, H).requires_grad_(True), _mk(T, H)
    idx = torch.rand(T, E, device="cuda").topk(k, dim=-1).indices
    p = None if probs is None else torch.rand(T, k, device="cuda").to(probs).requires_grad_(True)
    rows, order = M.permute(x, idx)
    assert torch.equal(rows, x.detach()[order // k])
    scaled = rows * 2.0
    out = M.unpermute(scaled, order, p, k, T)
    got = torch.autograd.grad(out, [x, scaled] + ([p] if p is not None else []), dout)
    xf = x.detach().float().requires_grad_(True)
    pf = None if p is None else p.detach().float().requires_grad_(True)
    sf = xf[order // k] * 2.0
    of = M.unpermute_reference(sf, order, pf, k, T * k)
    ref = torch.autograd.grad(of, [xf, sf] + ([pf] if p is not None else []), dout.float())
    for a, b in zip([out.detach(), *got], [of.detach(), *ref]):
        # dx passes three bf16 roundings (drows, its double, the sum), everything else one
        assert a.shape == b.shape and (a.float() - b).norm() <= 2 ** -7 * b.norm() + 1e-6


@pytest.mark.parametrize("T,K,heads,kv,D", [(256, 128, 2, 1, 128), (777, 264, 4, 2, 128), (300, 512, 4, 2, 64),
                                            (1000, 256, 3, 3, 128)])
@pytest.mark.parametrize("with_pos", [False, True])
def test_linear_rope_epilogue(T, K, heads, kv, D, with_pos):
    """Projection and rotation in one kernel against the two in fp32; the rounding of the projection is saved, so one
    bf16 rounding (2^-9) of the values and of the gradients remains. Heads past the rotated ones stay as they are."""
    from atorch_b200.ops import linear_rope, rope_reference, rope_tables

    torch.manual_seed(T)
    N = (heads + 2 * kv) * D
    x, w, dy = _mk(T, K).view(1, T, K).requires_grad_(True), (_mk(N, K) * 0.1).requires_grad_(True), _mk(T, N).view(1, T, N)
    pos = torch.randint(0, 2 * T, (1, T), device="cuda") if with_pos else None
    cos, sin = rope_tables(2 * T if with_pos else T, D, device="cuda")
    before = _lib.launch_count
    out = linear_rope(x, w, cos, sin, heads + kv, D, pos)
    rotated = (heads + kv) * D % 128 == 0 and N % 128 == 0
    assert _lib.launch_count - before == (1 if rotated else 2)
    got = torch.autograd.grad(out, [x, w], dy.clone())
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = rope_reference(xf @ wf.t(), cos, sin, heads + kv, D, pos)
    rg = torch.autograd.grad(ref, [xf, wf], dy.float())
    torch.cuda.synchronize()
    _lib.check_status(out.device)
    for a, b in zip([out.detach(), *got], [ref.detach(), *rg]):
        assert (a.float() - b).norm() <= 2 ** -7 * b.norm()


@pytest.mark.parametrize("T", [64, 256])
def test_linear_rope_leaves_the_incoming_gradient_alone(T):
    """The caller's gradient is read, not rotated in its place, in the fused kernel and in the two: two passes with the same
    tensor give the same bits. A layer may say that it is a temporary; the gradients are the same."""
    from atorch_b200.ops import linear_rope, rope_tables

    torch.manual_seed(T)
    x, w = _mk(T, 128).view(1, T, 128).requires_grad_(True), _mk(384, 128).requires_grad_(True)
    dy = _mk(T, 384).view(1, T, 384)
    kept = dy.clone()
    cos, sin = rope_tables(T, 128, device="cuda")
    out = linear_rope(x, w, cos, sin, 2, 128)
    res = [torch.autograd.grad(out, [x, w], dy, retain_graph=True) for _ in range(2)]
    assert torch.equal(dy, kept)
    res.append(torch.autograd.grad(linear_rope(x, w, cos, sin, 2, 128, inplace_grad=True), [x, w], dy))
    for other in res[1:]:
        assert all(torch.equal(a, b) for a, b in zip(res[0], other))


@pytest.mark.parametrize("sizes", [(256, 0, 1, 300), (77,), (0, 5, 511, 512, 513, 1)])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("N", [16, 272])
def test_grouped_gemm_swiglu_epilogue(sizes, trans_b, N):
    """The activation in the epilogue of the ragged launch: it rounds gate and up and uses the formula of the separate
    kernel, so results and gradients are the same bits; feature counts that are no multiple of the 128-column tile put
    columns of the other half, or of the next group, into the last tile."""
    from atorch_b200.ops import swiglu
    from atorch_b200.ops.moe import grouped_gemm, grouped_gemm_swiglu

    torch.manual_seed(sum(sizes))
    G, K = len(sizes), 192
    x = _mk(sum(sizes), K)
    w = (torch.randn(G, 2 * N, K, device="cuda") if trans_b else torch.randn(G, K, 2 * N, device="cuda")).bfloat16()
    dy = _mk(sum(sizes), N)
    res = []
    for f in (grouped_gemm_swiglu, lambda *a: swiglu(grouped_gemm(*a))):
        xs, ws = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
        before = _lib.launch_count
        y = f(xs, ws, sizes, trans_b)
        assert _lib.launch_count - before == (1 if f is grouped_gemm_swiglu else 2)
        y.backward(dy)
        with torch.no_grad():
            assert torch.equal(f(xs, ws, sizes, trans_b), y)
        res.append((y.detach(), xs.grad, ws.grad))
    torch.cuda.synchronize()
    _lib.check_status(x.device)
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n,k", [(1, 1), (31, 1), (32, 2), (1025, 1), (2051, 4), (8192, 4), (8193, 4)])
@pytest.mark.parametrize("E,ids", [(1, "one"), (8, "any"), (8, "last"), (256, "any"), (7, "bad")])
def test_route_sorts_stably(n, k, E, ids):
    """Counts, order, its inverse and the gathered rows are the ones of the stable sort, from one id to the largest
    number that the kernel takes and one above (the general path); ids out of range go to the end, uncounted."""
    from atorch_b200.ops import moe as M

    torch.manual_seed(n)
    x, dy = _mk(n, 24).requires_grad_(True), _mk(n * k, 24)
    idx = torch.full((n, k), E - 1) if ids in ("one", "last") else torch.randint(0, E, (n, k))
    own = n * k <= M.ROUTE_MAX_IDS
    if ids == "bad":
        if not own:
            pytest.skip("the general path refuses these")
        idx[::3] = E + 5
        idx[1::5] = -2
    counts, rows, order, slots = M.route(x, idx.cuda(), E)
    key = idx.flatten().clone()
    key[(key < 0) | (key >= E)] = E
    ref = torch.argsort(key, stable=True).cuda()
    assert torch.equal(order, ref) and torch.equal(counts.cpu(), torch.bincount(key, minlength=E + 1)[:E])
    assert (slots is not None) == own and torch.equal(rows, x.detach()[ref // k])
    if own:
        assert torch.equal(slots[order].cpu(), torch.arange(n * k, dtype=torch.int32))
    rows.backward(dy)
    back = torch.zeros(n, 24, device="cuda").index_add(0, ref // k, dy.float())
    assert (x.grad.float() - back).norm() <= 2 ** -8 * back.norm()


def test_routing_counts_may_be_changed_in_place():
    """A clamp of the counts (a capacity, a statistic) before the backward pass changes nothing else."""
    from atorch_b200.ops import moe as M

    torch.manual_seed(0)
    T, k, E = 40, 2, 4
    idx = torch.rand(T, E, device="cuda").topk(k, dim=-1).indices
    res = []
    for change in (False, True):
        torch.manual_seed(1)
        x, p = _mk(T, 64).requires_grad_(True), torch.rand(T, k, device="cuda").bfloat16().requires_grad_(True)
        counts, rows, order, slots = M.route(x, idx, E)
        out = M.unpermute(rows, order, p, k, T, slots)
        if change:
            counts.clamp_(max=3)
        res.append(torch.autograd.grad(out, [x, p], torch.ones_like(out)))
    assert all(torch.equal(a, b) for a, b in zip(*res))


def test_order_of_permute_may_be_changed_in_place():
    """What permute() and route() return is the caller's: the gradient of the rows does not come from it."""
    from atorch_b200.ops import moe as M

    torch.manual_seed(0)
    T, k, E = 40, 2, 4
    x, dy = _mk(T, 64).requires_grad_(True), _mk(T * k, 64)
    idx = torch.rand(T, E, device="cuda").topk(k, dim=-1).indices
    res = []
    for f in (lambda: M.permute(x, idx), lambda: M.route(x, idx, E)[1:3]):
        for change in (False, True):
            rows, order = f()
            if change:
                order.zero_()
            res.append(torch.autograd.grad(rows, x, dy)[0])
    assert all(torch.equal(res[0], r) for r in res[1:])


@pytest.mark.parametrize("probs", [None, torch.bfloat16])
def test_unpermute_keeps_the_rows_only_for_the_gradient_of_the_probabilities(probs):
    """Without such a gradient the rows are not kept: they may be changed in place after the call."""
    from atorch_b200.ops import moe as M

    torch.manual_seed(0)
    T, k, E, H = 40, 2, 4, 64
    order = torch.argsort(torch.rand(T, E, device="cuda").topk(k, dim=-1).indices.reshape(-1), stable=True)
    p = None if probs is None else torch.rand(T, k, device="cuda").to(probs)
    base, dout = _mk(T * k, H).requires_grad_(True), _mk(T, H)
    res = []
    for change in (False, True):
        rows = base * 1.0
        out = M.unpermute(rows, order, p, k, T)
        if change:
            rows.zero_()
        kept = [t for t in out.grad_fn.saved_tensors if t is not None and t.shape == rows.shape]
        assert not kept
        res.append(torch.autograd.grad(out, base, dout)[0])
    assert torch.equal(*res)


@pytest.mark.parametrize("probs_grad", [False, True])
def test_routed_rows_under_batched_gradients_and_tracing(probs_grad):
    """A batch of incoming gradients gives what one pass each gives (sums of k = 2 bf16 terms in another order: two
    roundings), and a trace holds operations, not the results of the traced inputs."""
    from torch.fx.experimental.proxy_tensor import make_fx

    from atorch_b200.ops import moe as M

    torch.manual_seed(0)
    T, k, E, H = 40, 2, 4, 64
    idx = torch.rand(T, E, device="cuda").topk(k, dim=-1).indices
    p = torch.rand(T, k, device="cuda").bfloat16().requires_grad_(probs_grad)

    def f(x, p):
        rows, order = M.permute(x, idx)
        routed, order2, slots = M.route(x, idx, E)[1:]
        return M.unpermute(rows, order, p, k, T), M.unpermute(routed, order2, p, k, T, slots)

    x = _mk(T, H).requires_grad_(True)
    wrt = [x, p] if probs_grad else [x]
    dout = _mk(3 * T, H).view(3, T, H)
    for out in f(x, p):
        got = torch.autograd.grad(out, wrt, dout, is_grads_batched=True, retain_graph=True)
        each = [torch.autograd.grad(out, wrt, d, retain_graph=True) for d in dout]
        for i, g in enumerate(got):
            ref = torch.stack([e[i] for e in each]).float()
            assert (g.float() - ref).norm() <= 2 ** -7 * ref.norm()
    with torch.no_grad():
        x2 = _mk(T, H)
        for pre in (False, True):
            traced = make_fx(f, pre_dispatch=pre)(x.detach(), p.detach())
            for a, b in zip(traced(x2, p.detach()), f(x2, p.detach())):
                assert (a.float() - b.float()).norm() <= 2 ** -7 * b.float().norm()


def test_expert_ids_out_of_range_are_refused():
    from atorch_b200.modules.moe import Grouped_GEMM_MoE

    with torch.device("cuda"):
        m = Grouped_GEMM_MoE(64, 64, 0.0, 4, 1, use_swiglu=True).bfloat16()
    x, p = _mk(8, 64), torch.ones(8, 1, device="cuda").bfloat16()
    for bad in (-1, 4):
        idx = torch.zeros(8, 1, dtype=torch.int64, device="cuda")
        idx[3] = bad
        with pytest.raises((AssertionError, RuntimeError, IndexError)):
            m(x, p, idx)


def test_routed_rows_under_transforms_and_second_derivatives():
    """What the row kernels hide from forward mode, vmap and a second derivative takes tensor operations: the same calls
    give what the plain composition gives (two bf16 roundings on either side)."""
    from atorch_b200.ops import moe as M

    torch.manual_seed(0)
    T, H, E, k = 37, 64, 4, 2
    x, p = _mk(T, H), torch.rand(T, k, device="cuda").bfloat16()
    idx = torch.randint(0, E, (T, k), device="cuda")

    def own(x, p):
        counts, rows, order, slots = M.route(x, idx, E)
        return M.unpermute(rows * rows, order, p, k, T, slots)

    def plain(x, p):
        return (x.unsqueeze(1) * x.unsqueeze(1) * p.unsqueeze(-1)).sum(1)

    def close(a, b):
        return (a.float() - b.float()).norm() <= 2 ** -6 * b.float().norm()

    res = []
    for f, dt in ((own, torch.bfloat16), (plain, torch.float32)):
        xs, ps = x.to(dt).requires_grad_(True), p.to(dt).requires_grad_(True)
        gx, gp = torch.autograd.grad(f(xs, ps).float().sum(), [xs, ps], create_graph=True)
        res.append(torch.autograd.grad(gx.float().square().sum() + gp.float().square().sum(), [xs, ps]))
    assert all(close(a, b) for a, b in zip(*res))
    tx, tp = torch.randn_like(x), torch.randn_like(p)
    a = torch.func.jvp(own, (x, p), (tx, tp))
    b = torch.func.jvp(plain, (x.float(), p.float()), (tx.float(), tp.float()))
    assert close(a[0], b[0]) and close(a[1], b[1])
    xs = torch.stack([x, tx])
    assert close(torch.func.vmap(own, (0, None))(xs, p), torch.func.vmap(plain, (0, None))(xs.float(), p.float()))


@pytest.mark.parametrize("sizes", [(1,), (64, 0, 63, 65, 129), (7,) * 17, (0, 300) + (5,) * 15])
@pytest.mark.parametrize("M,N", [(8, 264), (264, 8), (512, 256)])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.float32, True), (torch.float32, False)])
def test_gemm_k_groups(sizes, M, N, dtype, accumulate):
    """Weight gradients of row groups in one launch against one fp32 product each: last k-blocks of 1 to 64 rows, empty
    groups, more groups than a launch takes. Rows of the neighbours hold an infinity, which must not reach a group."""
    from atorch_b200.ops.gemm import gemm_k_groups, k_groups_ok

    torch.manual_seed(sum(sizes) + M)
    T, G = sum(sizes), len(sizes)
    a, b = _mk(T, M), _mk(T, N)
    a[0] = float("inf")
    b[0] = 1.0
    out = torch.randn(G, M, N, device="cuda").to(dtype) if accumulate else torch.full((G, M, N), float("nan"), device="cuda",
                                                                                      dtype=dtype)
    before = out.clone()
    assert k_groups_ok(a, b, out)
    gemm_k_groups(a, b, sizes, out, accumulate)
    torch.cuda.synchronize()
    _lib.check_status(out.device)
    r, first = 0, True
    for g, n in enumerate(sizes):
        ref = a[r: r + n].float().t() @ b[r: r + n].float() + (before[g].float() if accumulate else 0)
        if n and first:
            assert torch.isinf(out[g]).all()
            first = False
        else:
            # fp32 sums in another order, and one rounding of the output type
            tol = torch.finfo(dtype).eps + 2 * max(n, 1) ** 0.5 * 2 ** -23
            assert (out[g].float() - ref).norm() <= tol * max(ref.norm().item(), 1e-30)
        r += n


@pytest.mark.parametrize("sizes", [(64, 0, 63, 65, 129), (7,) * 17])
@pytest.mark.parametrize("M,N", [(8, 264), (264, 16), (512, 256)])
def test_gemm_k_groups_accumulates_in_bf16(sizes, M, N):
    """C += A_g^T B_g with a bf16 C, stored in 16-byte and in 32-byte pieces: one rounding of the fp32 sum (2^-9 of the result,
    twice that at the outside); groups without rows are left alone."""
    from atorch_b200.ops.gemm import gemm_k_groups, k_groups_ok

    torch.manual_seed(M)
    a, b = _mk(sum(sizes), M), _mk(sum(sizes), N)
    out = torch.randn(len(sizes), M, N, device="cuda").bfloat16()
    before = out.clone()
    assert k_groups_ok(a, b, out)
    gemm_k_groups(a, b, sizes, out, True)
    torch.cuda.synchronize()
    _lib.check_status(out.device)
    r = 0
    for g, n in enumerate(sizes):
        ref = before[g].double() + a[r: r + n].double().t() @ b[r: r + n].double()
        assert torch.equal(out[g], before[g]) if n == 0 else (out[g].double() - ref).norm() <= 2 ** -8 * ref.norm()
        r += n


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(256, 256, 128), (264, 264, 136), (8, 520, 1000), (1000, 2056, 192), (2560, 2560, 200)])
def test_gemm_two_pairs_per_tile(M, N, K, a_mn, b_mn):
    """A cluster of four CTAs per tile (tile_n = 512): the two halves of the reduction (unequal ones, of a single k-block, with a
    ragged end), more tiles than clusters, edges of rows and columns, every kind of output."""
    torch.manual_seed(M + N + K)
    a = _mk(K, M) if a_mn else _mk(M, K)
    b = _mk(K, N) if b_mn else _mk(N, K)
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    bias, res, c0 = _mk(1, N)[0], _mk(M, N), torch.randn(M, N, device="cuda")
    got = gemm(a, b, a_mn, b_mn, tile_n=512, kernel="2cta")
    both = gemm(a, b, a_mn, b_mn, tile_n=512, kernel="2cta", bias=bias, residual=res, alpha=0.5)
    acc = gemm(a, b, a_mn, b_mn, tile_n=512, kernel="2cta", out=c0.clone(), accumulate=True)
    torch.cuda.synchronize()
    _lib.check_status(a.device)
    for out, want, tol in ((got, ref, 2 ** -9), (both, 0.5 * ref + bias.double() + res.double(), 2 ** -9),   # one rounding to bf16
                           (acc, c0.double() + ref, 1e-5)):
        assert (out.double() - want).norm() <= tol * want.norm()


@pytest.mark.parametrize("T", [300, 512])
def test_fused_epilogues_with_two_pairs_per_tile(T):
    """SwiGLU and rotary epilogues on products of few tiles and a long reduction, which the rule gives two pairs per tile: gate
    and up, and the two sides of a rotation, meet in one thread again (heads of 128 and 64, columns that are not rotated, an
    edge inside a tile)."""
    from atorch_b200.ops import linear_rope, linear_swiglu
    from atorch_b200.ops.elementwise import rope_reference, rope_tables

    torch.manual_seed(T)
    K = 6144
    x, w = _mk(T, K), _mk(2 * 200, K) * 0.02
    g, u = (x.double() @ w.double().t()).to(torch.bfloat16).double().chunk(2, -1)
    act = linear_swiglu(x, w)
    want = torch.nn.functional.silu(g) * u
    assert (act.double() - want).norm() <= 2 ** -7 * want.norm()          # gate, up and the result are rounded to bf16
    for heads, kv, D in ((3, 2, 128), (4, 4, 64)):
        cos, sin = rope_tables(T, D, device="cuda")
        wq = _mk((heads + kv) * D, K) * 0.02
        got = linear_rope(x, wq, cos, sin, heads, D)
        want = rope_reference((x.double() @ wq.double().t()).float(), cos, sin, heads, D)
        torch.cuda.synchronize()
        _lib.check_status(x.device)
        assert (got.float() - want).norm() <= 2 ** -8 * want.norm()


@pytest.mark.parametrize("rows", [256, 777])
def test_kernels_that_start_early_wait_for_their_inputs(rows):
    """Every kernel of a chain reads what the one before wrote, and buffers are written again while they could still be read:
    the same bits with a synchronisation after each launch, without, and replayed from a graph."""
    from atorch_b200 import ops
    from atorch_b200.ops.flash import flash_attention

    torch.manual_seed(0)
    H = 512
    w = [(torch.randn(n, k, device="cuda") / k ** 0.5).bfloat16() for n, k in ((3 * H, H), (H, H), (4 * H, H), (H, 2 * H))]
    g = torch.ones(H, device="cuda").bfloat16()
    x0 = torch.randn(rows, H, device="cuda").bfloat16()
    x, act, out = torch.empty_like(x0), torch.empty(rows, 2 * H, device="cuda").bfloat16(), torch.empty_like(x0)
    bufs = [torch.empty(rows, n, device="cuda").bfloat16() for n in (3 * H, 4 * H)]

    def run(sync):
        x.copy_(x0)
        for _ in range(6):
            for step in (
                lambda: ops.gemm(ops.rms_norm(x, g, 1e-5), w[0], out=bufs[0]),
                lambda: out.copy_(flash_attention(*bufs[0].view(1, rows, 12, 128).split(4, 2), causal=True).view(rows, H)),
                lambda: ops.gemm(out, w[1], out=x, accumulate=True),
                lambda: ops.gemm(ops.rms_norm(x, g, 1e-5), w[2], out=bufs[1]),
                lambda: act.copy_(ops.swiglu(bufs[1])),
                lambda: ops.gemm(act, w[3], out=x, accumulate=True),
            ):
                step()
                if sync:
                    torch.cuda.synchronize()
        return x.clone()

    with torch.no_grad():
        want = run(True)
        assert all(torch.equal(run(False), want) for _ in range(20))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = run(False)
        for _ in range(5):
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(got, want)
    assert bool(torch.isfinite(want).all())


@pytest.mark.parametrize("kind", ["one wave", "many tiles", "two pairs per tile", "accumulate", "attention", "attention backward"])
def test_kernel_behind_an_error_stores_nothing(kind):
    """The kernel in front records an error (the status word is the last element that it writes) after the kernel behind has
    started early: the kernel behind stores nothing, and no wait of it runs out. With a clear word it stores everything."""
    torch.manual_seed(0)
    L, st = _lib.lib(), _lib.stream()
    a = torch.ones(4096, 8192, device="cuda", dtype=torch.bfloat16)
    front = torch.zeros(4096, 4096, device="cuda", dtype=torch.bfloat16)
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    if kind.startswith("attention"):
        B, S, H, D = 2, 640, 16, 128
        q, k, v, do, o = (rnd(B, S, H, D) for _ in range(5))
        lse, delta = torch.zeros(B, H, S, device="cuda"), torch.zeros(B * H * S, device="cuda")
        outs = [torch.zeros_like(q) for _ in range(3)]
        dims = (0, 0, B, S, S, H, H, H * D, H * D, H * D)

        def launch(status):
            p = [t.data_ptr() for t in outs]
            if kind == "attention":
                return L.atb_flash_fwd_v2(q.data_ptr(), k.data_ptr(), v.data_ptr(), p[0], lse.data_ptr(), *dims, 1, D ** -0.5,
                                          st, status, D, 0)
            return L.atb_flash_bwd_split(do.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                                         lse.data_ptr(), delta.data_ptr(), *p, *dims, H * D, H * D, H * D, 1, D ** -0.5, st,
                                         status, 1, D)
        outs_written = outs[:1] if kind == "attention" else outs
    else:
        M, N, K = {"one wave": (512, 512, 512), "accumulate": (777, 520, 256)}.get(kind, (4096, 4096, 1024))
        x, w, c = rnd(M, K), rnd(N, K), torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        outs_written = [c]

        def launch(status):
            return L.atb_gemm_bf16_2cta(x.data_ptr(), w.data_ptr(), c.data_ptr(), 0, M, N, K, K, K, N, 0, 0, 0,
                                        int(kind == "accumulate"), 1.0, 512 if kind == "two pairs per tile" else 0, 0, 0, 0, st,
                                        status)
    word = front.view(torch.int32)[-1, -1:]
    for _ in range(3):
        front.zero_()
        gemm(a, a[:4096], out=front)
        assert launch(word.data_ptr()) == 0
        torch.cuda.synchronize()
        assert front.view(torch.int32)[-1, -1].item() == 0x46004600      # 8192 twice: what the product wrote, no error code
        assert not any(bool(t.any()) for t in outs_written)
    clear = torch.zeros(1, device="cuda", dtype=torch.int32)
    assert launch(clear.data_ptr()) == 0
    torch.cuda.synchronize()
    assert clear.item() == 0 and all(bool(t.any()) for t in outs_written)


def test_gate_behind_an_error_does_not_wait():
    """Rows that have not arrived are not waited for once an error has been recorded, and nothing is stored."""
    import ctypes
    import time

    M, N, K = 512, 1024, 512
    x, w = _mk(M, K), _mk(N, K)
    c = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    flags = torch.zeros(8, device="cuda", dtype=torch.int32)
    status = torch.full((1,), 4, device="cuda", dtype=torch.int32)
    ll, p = ctypes.c_longlong, lambda t: ctypes.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    t0 = time.time()
    for _ in range(4):
        assert _lib.lib().atb_gemm_bf16_2cta_wgather(p(x), p(w), p(c), M, N, K, ll(K), ll(K), ll(N), p(flags),
                                                     ctypes.c_uint(1), 128, 256, _lib.stream_ptr(), p(status)) == 0
    torch.cuda.synchronize()
    assert time.time() - t0 < 1.0                # the limit of one wait is 2 s
    assert not bool(c.any()) and status.item() == 4
    status.zero_()
    flags.fill_(1)
    assert _lib.lib().atb_gemm_bf16_2cta_wgather(p(x), p(w), p(c), M, N, K, ll(K), ll(K), ll(N), p(flags), ctypes.c_uint(1),
                                                 128, 256, _lib.stream_ptr(), p(status)) == 0
    _check(c, x.float() @ w.float().t(), K)


def test_launch_with_a_limit_leaves_the_other_sms_free():
    """20 CTAs for some milliseconds and a product of the same stream behind them: one of another stream, which needs SMs to
    itself, ends long before they do."""
    a, small = _mk(8192, 8192), _mk(2048, 2048)
    side = torch.cuda.Stream()
    first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    gemm(a, a, max_ctas=20)
    gemm(small, small)
    with torch.cuda.stream(side):
        gemm(small, small)
    torch.cuda.synchronize()
    gemm(a, a, max_ctas=20)
    gemm(small, small)
    with torch.cuda.stream(side):
        gemm(small, small)
        first.record()
    last.record()
    torch.cuda.synchronize()
    _lib.check_status(a.device)
    assert first.elapsed_time(last) > 1.0


def test_shared_tiles_beside_another_kernel():
    """Two pairs per tile, six tiles per cluster, while a launch of another stream holds 24 SMs: the clusters that fit share the
    tiles. With a fixed share of six, those that start when the first ones end double the time."""
    held, side = _mk(8192, 8192), torch.cuda.Stream()
    x, w = _mk(37 * 256, 2048), _mk(6 * 256, 2048)
    out, ms = torch.empty(37 * 256, 6 * 256, device="cuda", dtype=torch.bfloat16), {}
    for hold in (False, True, False, True):
        torch.cuda.synchronize()
        if hold:
            with torch.cuda.stream(side):
                gemm(held, held, max_ctas=24)
        first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        out.fill_(float("nan"))
        torch.cuda._sleep(400000)            # the launch of the other stream has its SMs
        first.record()
        gemm(x, w, out=out, tile_n=512)
        last.record()
        torch.cuda.synchronize()
        ms[hold] = first.elapsed_time(last)
        _check(out, x.float() @ w.float().t(), 2048)
    _lib.check_status(x.device)
    assert ms[True] < 1.5 * ms[False], ms


def test_adding_to_fp32_costs_reading_it():
    """A product that adds to an fp32 output reads and writes it, one that only writes it moves half as much: with room for the
    lines of the output in the L1 cache twice to 2.3 times the time, without it three times."""
    x, w, out, us = _mk(4096, 64), _mk(11008, 64), torch.zeros(4096, 11008, device="cuda"), {}
    for add in (False, True) * 6:
        first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(200000)
        first.record()
        gemm(x, w, out=out, accumulate=add)
        last.record()
        torch.cuda.synchronize()
        us[add] = min(us.get(add, 1e9), 1e3 * first.elapsed_time(last))
    assert us[True] < 2.6 * us[False], us


@pytest.mark.parametrize("rows", [300, 2048])
def test_early_starts_forward_backward_and_across_streams(rows):
    """A layer and its gradients, with its products that two pairs share, and a product of another stream behind an event: the
    same bits with a synchronisation after every operator of both passes and without."""
    from atorch_b200 import ops
    from atorch_b200.ops.flash import flash_attention_qkv

    torch.manual_seed(1)
    H, F, side = 1024, 6144, torch.cuda.Stream()
    w = [(torch.randn(n, k, device="cuda") / k ** 0.5).bfloat16().requires_grad_() for n, k in ((3 * H, H), (H, H), (2 * F, H), (H, F))]
    g = torch.ones(H, device="cuda").bfloat16().requires_grad_()
    x0, dy = torch.randn(1, rows, H, device="cuda").bfloat16().requires_grad_(), torch.randn(1, rows, H, device="cuda").bfloat16()
    cos, sin = ops.rope_tables(rows, 128, 10000.0, "cuda")

    def run(sync):
        def mark(t):
            if sync:
                torch.cuda.synchronize()
                t.register_hook(lambda d: torch.cuda.synchronize())
            return t

        qkv = mark(ops.rope(mark(ops.linear(mark(ops.rms_norm(x0, g, 1e-5)), w[0])), cos, sin, 16, 128))
        a = mark(flash_attention_qkv(qkv.view(1, rows, 24, 128), 8))
        x = mark(ops.linear(a.view(1, rows, H), w[1], residual=x0))
        act = mark(ops.swiglu(mark(ops.linear(mark(ops.rms_norm(x, g, 1e-5)), w[2]))))
        y = mark(ops.linear(act, w[3], residual=x))
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            z = ops.gemm(y.detach().view(rows, H), y.detach().view(rows, H))
        grads = torch.autograd.grad(y, (x0, g, *w), dy)
        torch.cuda.current_stream().wait_stream(side)
        with torch.no_grad():
            z = ops.gemm(z[:256], z[:256])
        torch.cuda.synchronize()
        return (y.detach(), z, *grads)

    want = run(True)
    assert all(bool(torch.isfinite(t).all()) for t in want)
    for _ in range(8):
        for a, b in zip(run(False), want):
            assert torch.equal(a, b)
    _lib.check_status(x0.device)


@pytest.mark.parametrize("tile_n", [256, 512])
def test_graphs_of_one_stream_replayed_beside_each_other(tile_n):
    """Two graphs captured on a stream that has run the same products before, replayed on two other streams while that one
    runs them too: each result is whole."""
    side, streams = torch.cuda.Stream(), [torch.cuda.Stream() for _ in range(2)]
    x, w = [_mk(4096, 512) for _ in range(3)], _mk(4096, 512)
    outs = [torch.empty(4096, 4096, device="cuda", dtype=torch.bfloat16) for _ in x]

    def run(i):
        for _ in range(8):
            gemm(x[i], w, out=outs[i], tile_n=tile_n)

    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        run(2)
    torch.cuda.synchronize()
    graphs = [torch.cuda.CUDAGraph() for _ in streams]
    for i, g in enumerate(graphs):
        with torch.cuda.graph(g, stream=side):
            run(i)
    want = [gemm(t, w, tile_n=tile_n) for t in x]
    for _ in range(20):
        for o in outs:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(side):
            run(2)
        torch.cuda.synchronize()
        for o, t in zip(outs, want):
            assert torch.equal(o, t)
    _lib.check_status(w.device)
