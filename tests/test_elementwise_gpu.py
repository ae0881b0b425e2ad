"""Row / elementwise sm_100a kernels against fp32 PyTorch references."""
import pytest
import torch

from atorch_b200 import ops

pytestmark = pytest.mark.gpu


def _close(a, b, rtol=2e-2, atol=2e-2):
    torch.cuda.synchronize()
    assert torch.allclose(a.float(), b.float(), rtol=rtol, atol=atol), (a.float() - b.float()).abs().max().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,N", [(1, 64), (37, 1000), (513, 4096), (64, 8192)])
def test_rmsnorm_fwd_bwd(M, N, dtype):
    torch.manual_seed(0)
    x = torch.randn(M, N, device="cuda", dtype=dtype, requires_grad=True)
    w = (1 + 0.1 * torch.randn(N, device="cuda")).to(dtype).requires_grad_()
    dy = torch.randn(M, N, device="cuda", dtype=dtype)
    y = ops.rms_norm(x, w, 1e-5)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    yr.backward(dy.float())
    tol = 1e-4 if dtype == torch.float32 else 3e-2
    _close(y, yr, tol, tol)
    _close(x.grad, xr.grad, tol, tol)
    _close(w.grad, wr.grad, tol, tol * max(1.0, M ** 0.5))


def test_rmsnorm_residual_and_main_grad():
    torch.manual_seed(1)
    M, N = 200, 2048
    x = torch.randn(M, N, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(M, N, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.ones(N, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w.main_grad = torch.zeros(N, device="cuda", dtype=torch.float32)
    y, s = ops.rms_norm(x, w, 1e-5, residual=r)
    (y.float().sum() + 2 * s.float().sum()).backward()
    xr = (x.detach().float() + r.detach().float()).to(torch.bfloat16).float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    (yr.sum() + 2 * xr.sum()).backward()
    _close(s, xr)
    _close(y, yr)
    _close(x.grad, xr.grad, 3e-2, 3e-2)
    assert torch.equal(x.grad, r.grad)
    assert w.grad is None
    _close(w.main_grad, wr.grad, 3e-2, 0.5)


@pytest.mark.parametrize("M,N", [(33, 768), (128, 1024)])
def test_layernorm_fwd_bwd(M, N):
    torch.manual_seed(2)
    x = torch.randn(M, N, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16().requires_grad_()
    b = (0.1 * torch.randn(N, device="cuda")).bfloat16().requires_grad_()
    dy = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    y = ops.layer_norm(x, w, b, 1e-5)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.layer_norm(xr, (N,), wr, br, 1e-5)
    yr.backward(dy.float())
    _close(y, yr, 3e-2, 3e-2)
    _close(x.grad, xr.grad, 3e-2, 3e-2)
    _close(w.grad, wr.grad, 3e-2, 0.3)
    _close(b.grad, br.grad, 3e-2, 0.3)


def test_rope_matches_reference_and_is_orthogonal():
    torch.manual_seed(3)
    B, S, nq, nkv, d = 2, 128, 4, 2, 128
    W = (nq + 2 * nkv) * d
    x = torch.randn(B, S, W, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    cos, sin = ops.rope_tables(S, d, device="cuda")
    y = ops.rope(x, cos, sin, nq + nkv, d)
    ref = ops.rope_reference(x.detach(), cos, sin, nq + nkv, d)
    _close(y, ref, 1e-2, 1e-2)
    assert torch.equal(y[..., (nq + nkv) * d:], x[..., (nq + nkv) * d:])
    dy = torch.randn_like(y)
    y.backward(dy)
    refg = ops.rope_reference(dy, cos, sin, nq + nkv, d, backward=True)
    _close(x.grad, refg, 1e-2, 1e-2)
    pos = torch.randint(0, S, (B * S,), device="cuda", dtype=torch.int32)
    y2 = ops.rope(x.detach(), cos, sin, nq, d, positions=pos)
    _close(y2, ops.rope_reference(x.detach(), cos, sin, nq, d, positions=pos), 1e-2, 1e-2)


def test_rope_in_place_matches_out_of_place():
    torch.manual_seed(5)
    B, S, nq, nkv, d = 2, 128, 4, 4, 128
    W = (nq + 2 * nkv) * d
    x = torch.randn(B, S, W, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    cos, sin = ops.rope_tables(S, d, device="cuda")
    ref = ops.rope(x, cos, sin, nq + nkv, d)
    dy = torch.randn_like(ref)
    ref.backward(dy.clone())
    g_ref, x.grad = x.grad.clone(), None
    h = x * 1.0                                  # a non-leaf that nothing else reads
    y = ops.rope(h, cos, sin, nq + nkv, d, inplace=True)
    assert y.data_ptr() == h.data_ptr()          # rotated where it is
    assert torch.equal(y, ref)
    y.backward(dy.clone())
    assert torch.equal(x.grad, g_ref)
    # a leaf is never overwritten
    z = ops.rope(x, cos, sin, nq + nkv, d, inplace=True)
    assert z.data_ptr() != x.data_ptr()


def test_swiglu_fwd_bwd():
    torch.manual_seed(4)
    gu = torch.randn(300, 2 * 1376, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(300, 1376, device="cuda", dtype=torch.bfloat16)
    y = ops.swiglu(gu)
    y.backward(dy)
    gr = gu.detach().float().requires_grad_()
    yr = torch.nn.functional.silu(gr[:, :1376]) * gr[:, 1376:]
    yr.backward(dy.float())
    _close(y, yr)
    _close(gu.grad, gr.grad, 3e-2, 3e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [32000, 1003])
@pytest.mark.parametrize("smooth,z", [(0.0, 0.0), (0.1, 1e-4)])
def test_cross_entropy(V, dtype, smooth, z):
    torch.manual_seed(5)
    rows = 257
    Vp = (V + 7) // 8 * 8
    buf = torch.randn(rows, Vp, device="cuda", dtype=dtype) * 2
    logits = buf[:, :V].detach().requires_grad_()
    labels = torch.randint(0, V, (rows,), device="cuda")
    labels[::7] = -100
    loss = ops.cross_entropy(logits, labels, label_smoothing=smooth, lse_square_scale=z)
    w = torch.rand(rows, device="cuda")
    (loss * w).sum().backward()
    lr = logits.detach().float().requires_grad_()
    ref = ops.cross_entropy_reference(lr, labels, -100, smooth, z)
    (ref * w).sum().backward()
    _close(loss, ref, 1e-3, 1e-3)
    tol = 1e-5 if dtype == torch.float32 else 1e-2
    _close(logits.grad, lr.grad, tol, tol)


def test_adamw_and_agd_steps():
    torch.manual_seed(6)
    n = 100003
    for gd in (torch.bfloat16, torch.float32):
        master = torch.randn(n, device="cuda")
        m, v = torch.zeros_like(master), torch.zeros_like(master)
        lp = torch.empty(n, device="cuda", dtype=torch.bfloat16)
        mr, m2, v2 = master.clone(), m.clone(), v.clone()
        for step in range(1, 4):
            g = torch.randn(n, device="cuda").to(gd)
            ops.adamw_step(master, m, v, g, lp, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, grad_scale=0.5)
            ops.adamw_reference(mr, m2, v2, g, None, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, grad_scale=0.5)
        _close(master, mr, 1e-5, 1e-5)
        _close(lp, mr.bfloat16(), 1e-2, 1e-2)
        master = torch.randn(n, device="cuda")
        m, v = torch.zeros_like(master), torch.zeros_like(master)
        mr, m2, v2 = master.clone(), m.clone(), v.clone()
        for step in range(1, 4):
            g = torch.randn(n, device="cuda").to(gd)
            ops.agd_step(master, m, v, g, lp, 1e-2, 0.9, 0.999, 1e-5, 0.1, step)
            ops.agd_reference(mr, m2, v2, g, None, 1e-2, 0.9, 0.999, 1e-5, 0.1, step)
        _close(master, mr, 1e-4, 1e-4)


def test_sum_squares_and_outer_sgd():
    torch.manual_seed(7)
    x = torch.randn(1 << 20, device="cuda")
    ref = x.double().pow(2).sum().item()
    assert abs(ops.sum_squares(x).item() - ref) < 2e-6 * ref
    n = 5000
    synced, buf, pg = torch.randn(n, device="cuda"), torch.zeros(n, device="cuda"), torch.randn(n, device="cuda")
    p = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    s2, b2 = synced.clone(), buf.clone()
    for i in range(3):
        ops.outer_sgd_step(synced, buf, pg, p, 0.7, 0.9, True, i == 0)
        ops.outer_sgd_reference(s2, b2, pg, None, 0.7, 0.9, True, i == 0)
    _close(synced, s2, 1e-5, 1e-5)
    _close(p, s2.bfloat16(), 1e-2, 1e-2)


def test_bias_gather_add():
    torch.manual_seed(8)
    inp = torch.randn(100, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    bias = torch.randn(8, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    idx = torch.randint(0, 8, (100,), device="cuda")
    out = ops.bias_gather_add(inp, bias, idx)
    _close(out, ops.bias_gather_add_reference(inp.detach(), bias.detach(), idx))
    out.sum().backward()
    cnt = torch.bincount(idx, minlength=8).float()
    _close(bias.grad, cnt[:, None].expand(8, 256), 1e-2, 1e-2)


def test_rmsnorm_carry_adds_the_residual_gradient_in_the_kernel():
    """``carry=True`` hands x back for the residual path: no copy, and the gradient through it is added inside the
    backward kernel. Same numbers as the plain form plus autograd's own add."""
    torch.manual_seed(8)
    x = torch.randn(512, 4096, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(4096, device="cuda", dtype=torch.bfloat16)
    dy, dres = torch.randn_like(x), torch.randn_like(x)
    xa, wa = x.clone().requires_grad_(), w.clone().requires_grad_()
    h = xa * 1.0
    y, carried = ops.rms_norm(h, wa, 1e-5, carry=True)
    assert carried.data_ptr() == h.data_ptr() and torch.equal(carried, h)
    torch.autograd.backward([y, carried], [dy, dres])
    xb, wb = x.clone().requires_grad_(), w.clone().requires_grad_()
    y2 = ops.rms_norm(xb, wb, 1e-5)
    assert torch.equal(y, y2)
    y2.backward(dy)
    ref = xb.grad.float() + dres.float()
    _close(xa.grad, ref, 2e-2, 2e-2)
    assert torch.equal(wa.grad, wb.grad)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 3, 8, 4097, 148 * 4 * 256 * 8 * 4, (1 << 22) + 5])
def test_sum_squares_lengths_and_alignment(n, dtype):
    """Whole and partial 16-byte pieces, one and several rounds of the grid, and a start that is not 16-byte aligned.
    Every element's square is rounded once and added in a chain of at most a few hundred terms: relative error below
    2^-24 sqrt(300) on average, 1e-5 at the outside."""
    torch.manual_seed(n)
    buf = torch.randn(n + 1, device="cuda").to(dtype)
    for x in (buf[:n], buf[1:]):
        ref = x.double().square().sum()
        assert abs(ops.sum_squares(x).double() - ref) <= 1e-5 * ref


@pytest.mark.parametrize("M,N,dtype", [(1, 2048, torch.bfloat16), (297, 8, torch.float16), (1187, 2048, torch.bfloat16),
                                       (1187, 2056, torch.bfloat16), (600, 4104, torch.float16),
                                       (300, 8192, torch.bfloat16), (1187, 2048, torch.float32),
                                       (599, 4096, torch.float32), (300, 8192, torch.float32)])
@pytest.mark.parametrize("layernorm", [False, True])
def test_norm_backward_row_pairs(M, N, dtype, layernorm):
    """Backward kernels at the edges of their row pairs (odd chunks, empty chunks, one row) and of each row length, with
    the residual gradient, against 64 bits. Inputs are exact in both, so what is left in dx is its own rounding (eps / 2) and the
    fp32 sums (a few N-term sums, taken as 16 times the fp32 eps); dw is rounded once more on its way to the parameter."""
    from atorch_b200 import _lib

    torch.manual_seed(M + N)
    x, dy, dres = (torch.randn(M, N, device="cuda").to(dtype) for _ in range(3))
    w = (1 + 0.1 * torch.randn(N, device="cuda")).to(dtype)
    xd, wd, dyd = x.double(), w.double(), dy.double()
    mean = xd.mean(-1) if layernorm else torch.zeros(M, device="cuda", dtype=torch.float64)
    rstd = ((xd - mean[:, None]).pow(2).mean(-1) + 1e-5).rsqrt()
    mean, rstd = mean.float(), rstd.float()
    xh = (xd - mean.double()[:, None]) * rstd.double()[:, None]
    g = dyd * wd
    ref = (g - xh * (g * xh).mean(-1, keepdim=True) - (g.mean(-1, keepdim=True) if layernorm else 0)) * rstd.double()[:, None]
    ref = ref + dres.double()
    parts = _lib.lib().atb_norm_bwd_parts(M)
    dx, pw, pb = torch.full_like(x, float("nan")), torch.full((parts, N), float("nan"), device="cuda"), None
    pb = torch.full_like(pw, float("nan")) if layernorm else None
    rc = _lib.lib().atb_norm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                 dres.data_ptr(), dx.data_ptr(), pw.data_ptr(), _lib.addr(pb), parts, M, N, int(layernorm),
                                 _lib.DT[dtype], _lib.stream())
    assert rc == 0
    eps32 = torch.finfo(torch.float32).eps
    assert (dx.double() - ref).norm() <= (torch.finfo(dtype).eps / 2 + 16 * eps32) * ref.norm()
    dw = (dyd * xh).sum(0)
    assert (pw.double().sum(0) - dw).norm() <= 16 * eps32 * max(1.0, M ** 0.5) * dw.norm()
    if layernorm:
        assert (pb.double().sum(0) - dyd.sum(0)).norm() <= 16 * eps32 * max(1.0, M ** 0.5) * dyd.sum(0).norm()


@pytest.mark.parametrize("T,V,H,out_dtype,accumulate,ids_of", [
    (1, 1, 8, torch.bfloat16, False, "uniform"),
    (777, 1000, 520, torch.bfloat16, True, "uniform"),
    (8193, 32000, 256, torch.float32, True, "uniform"),
    (4100, 151937, 64, torch.bfloat16, False, "uniform"),       # ranges of 1024 rows, the last one ragged
    (5000, 149, 1032, torch.float32, False, "padding"),         # most tokens on one row: a block sums it
    (300, 31, 512, torch.bfloat16, True, "edge"),               # 63 to 66 tokens a row
])
def test_embedding_gradient(T, V, H, out_dtype, accumulate, ids_of):
    from atorch_b200.ops.embedding import embedding_grad

    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, V, (T,), generator=g)
    if ids_of == "padding":
        ids[torch.rand(T, generator=g) < 0.8] = V - 1
    elif ids_of == "edge":
        ids = torch.cat([torch.full((n,), i * 7) for i, n in enumerate((63, 64, 65, 66, 42))])[torch.randperm(T, generator=g)]
    dy = torch.randn(T, H, generator=g).bfloat16()
    old = torch.randn(V, H, generator=g).to(out_dtype)
    out = old.cuda() if accumulate else torch.full((V, H), float("nan"), dtype=out_dtype, device="cuda")
    embedding_grad(dy.cuda(), ids.cuda(), out, accumulate)
    want = (old.double() if accumulate else torch.zeros(V, H, dtype=torch.float64)).index_add(0, ids, dy.double())
    size = (old.double().abs() if accumulate else torch.zeros(V, H, dtype=torch.float64)).index_add(0, ids, dy.double().abs())
    n = torch.bincount(ids, minlength=V).max().item() + 1
    # n fp32 additions and one rounding to the output type
    bound = size * n * 2.0 ** -23 + (want.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0.0)
    assert bool(((out.double().cpu() - want).abs() <= bound).all())
    again = old.cuda() if accumulate else torch.empty_like(out)
    assert torch.equal(embedding_grad(dy.cuda(), ids.cuda(), again, accumulate), out)     # same bits whatever the timing


def test_embedding_module_gradient_and_fallbacks():
    m = torch.nn.Embedding(300, 64).cuda().bfloat16()
    ids = torch.randint(0, 300, (3, 50), device="cuda")
    w = torch.randn(3, 50, 64, device="cuda")
    out = ops.embedding(m, ids)
    (out.float() * w).sum().backward()
    got, m.weight.grad = m.weight.grad, None
    assert torch.equal(out, torch.nn.functional.embedding(ids, m.weight))
    dy = w.bfloat16().double().view(-1, 64)
    want = torch.zeros(300, 64, dtype=torch.float64, device="cuda").index_add(0, ids.view(-1), dy)
    # one rounding of an fp32 sum (the library adds up in bf16 where there are few tokens)
    torch.testing.assert_close(got.double(), want, rtol=2.0 ** -8, atol=1e-6)
    m.weight.grad = None
    m.weight.main_grad = torch.ones(300, 64, device="cuda")
    (ops.embedding(m, ids).float() * w).sum().backward()
    assert m.weight.grad is None and m.weight.grad_added_to_main_grad
    torch.testing.assert_close(m.weight.main_grad.double() - 1, want, rtol=0.0, atol=2.0 ** -20)     # fp32 sums below 8
    seen = []
    m.register_forward_hook(lambda *a: seen.append(1))
    ops.embedding(m, ids)
    assert seen == [1]


@pytest.mark.parametrize("dtype,off", [(torch.bfloat16, 0), (torch.float32, 1), (torch.float64, 0)])
def test_embedding_into_an_untouched_buffer(dtype, off):
    """A gradient buffer that nothing has been written to is overwritten, also one that the kernels do not take."""
    m = torch.nn.Embedding(300, 64).cuda().bfloat16()
    ids = torch.randint(0, 300, (150,), device="cuda")
    m.weight.main_grad = torch.full((300 * 64 + off,), float("nan"), dtype=dtype, device="cuda")[off:].view(300, 64)
    m.weight._atb_first = True
    w = torch.randn(150, 64, device="cuda").bfloat16()
    ops.embedding(m, ids).backward(w)
    want = torch.zeros(300, 64, dtype=torch.float64, device="cuda").index_add(0, ids, w.double())
    torch.testing.assert_close(m.weight.main_grad.double(), want, rtol=2.0 ** -8, atol=1e-6)     # one rounding to bf16
    assert m.weight._atb_first is False and m.weight.grad_added_to_main_grad


def test_embedding_leaves_watched_calls_to_the_module():
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    m = torch.nn.Embedding(300, 64).cuda().bfloat16()
    ids = torch.randint(0, 300, (150,), device="cuda")
    node = lambda: type(ops.embedding(m, ids).grad_fn).__name__
    own = node()
    assert own == "_EmbeddingFnBackward"
    with torch.device("cuda"):          # says where tensors are made, looks at nothing
        assert node() == own
    for mode in (Dispatch(), Function()):
        with mode:
            assert node() != own
    seen = []
    m._compiled_call_impl = lambda *a: seen.append(a) or m.forward(*a)      # what module.compile() sets
    assert node() != own and len(seen) == 1


@pytest.mark.parametrize("out_dtype,accumulate", [(torch.bfloat16, False), (torch.float32, True)])
@pytest.mark.parametrize("counts,V,H", [
    ((512,), 1, 8),                                        # the most that one block sums, and one more
    ((513,), 2, 520),
    ((1, 511, 512, 513, 1023, 1024, 1025, 0, 200, 600, 1400, 1), 40, 264),    # rows that begin and end everywhere in a part
    ((600, 0, 600, 600, 5, 6000), 3000, 1032),
])
def test_embedding_gradient_of_long_rows(counts, V, H, out_dtype, accumulate):
    from atorch_b200.ops.embedding import embedding_grad

    g = torch.Generator().manual_seed(sum(counts))
    rows = torch.randperm(V, generator=g)[: len(counts)].sort().values
    ids = torch.repeat_interleave(rows, torch.tensor(counts[: len(rows)]))
    ids = ids[torch.randperm(ids.numel(), generator=g)]
    dy = torch.randn(ids.numel(), H, generator=g).bfloat16()
    old = torch.randn(V, H, generator=g).to(out_dtype)
    out = old.cuda() if accumulate else torch.full((V, H), float("nan"), dtype=out_dtype, device="cuda")
    embedding_grad(dy.cuda(), ids.cuda(), out, accumulate)
    want = (old.double() if accumulate else torch.zeros(V, H, dtype=torch.float64)).index_add(0, ids, dy.double())
    size = (old.double().abs() if accumulate else torch.zeros(V, H, dtype=torch.float64)).index_add(0, ids, dy.double().abs())
    # as many fp32 additions as a row has tokens, and one rounding to the output type
    bound = size * (max(counts) + 1) * 2.0 ** -23 + (want.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0.0)
    assert bool(((out.double().cpu() - want).abs() <= bound).all())
    again = old.cuda() if accumulate else torch.empty_like(out)
    assert torch.equal(embedding_grad(dy.cuda(), ids.cuda(), again, accumulate), out)


def test_embedding_gradient_time_does_not_depend_on_the_ids():
    """A row with most of the tokens (padding), and a table of few rows, take about as long as tokens spread over a large one."""
    from atorch_b200.ops.embedding import embedding_grad

    T, H, us = 65536, 1024, {}
    dy = torch.randn(T, H, device="cuda").bfloat16()
    for name, V, ids in (("spread", 32000, torch.randint(0, 32000, (T,), device="cuda")),
                         ("one", 32000, torch.zeros(T, dtype=torch.int64, device="cuda")),
                         ("few", 256, torch.randint(0, 256, (T,), device="cuda"))):
        out = torch.zeros(V, H, device="cuda", dtype=torch.bfloat16)
        for _ in range(5):
            first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda._sleep(200000)
            first.record()
            embedding_grad(dy, ids, out, True)
            last.record()
            torch.cuda.synchronize()
            us[name] = min(us.get(name, 1e9), 1e3 * first.elapsed_time(last))
    assert us["one"] < 3 * us["spread"] and us["few"] < 3 * us["spread"], us
