"""bf16 GEMM on the tcgen05 tensor cores and the autograd ``linear`` built on it.

``gemm`` computes ``C (+)= alpha * op(A) @ op(B)^T (+ bias)`` with either operand stored K-major or
MN-major, so that the forward, dgrad and wgrad products of a linear layer all read their operands
as they lie in memory. On a CPU-only machine the same function evaluates the product with PyTorch
(the reference implementation that the GPU tests compare against).

``linear`` is the drop-in for ``torch.nn.functional.linear`` used by every projection of the models
in this package. Its backward accumulates the weight gradient straight into ``weight.main_grad``
when the parameter carries such a buffer (the flat gradient buffers of the sharded data-parallel
engines), which removes the separate gradient tensor and the accumulate pass.

Reference counterpart: cuBLAS behind ``nn.Linear`` (atorch/modules/distributed_modules/layers.py:117-151).
"""
from __future__ import annotations

import ctypes
import os
from typing import Optional

import torch

from .. import _lib
from .function import call


# CTA-pair kernel (tcgen05 cta_group::2, 256x256 tiles) for problems with M, N >= 256
PAIR_KERNEL_DEFAULT = os.environ.get("ATB_GEMM_PAIR", "1") == "1"


def _pitch(t: torch.Tensor) -> int:
    return t.stride(0) if t.dim() == 2 else t.shape[-1]


def _sizes_ok(a, b, M, N, K, a_mn, b_mn, out, groups, bias, residual) -> bool:
    """Whether the kernels take these sizes. They store 8 columns at a time and load 16-byte pieces along the dim in
    which an operand is contiguous; the other dim of an operand may have any length (rows of A in the forward product
    and in dgrad, the reduction dim in wgrad: the tensor maps read zeros past the end), which is where the token count
    of a ragged batch goes. Evaluating a 1.3B model of 8 layers on 777 tokens (25 such products) takes 1.8 ms of GPU
    time with them here, 11.3 ms with them on the fp32 fallback."""
    if N % 8 == 0 and K % 8 == 0 and M % 8 == 0:
        return True
    if N % 8 or (a_mn and M % 8) or (K % 8 and not (a_mn and b_mn)) or groups is not None:
        return False
    if residual is not None and (out.dtype != torch.bfloat16 or residual.dtype != torch.bfloat16
                                 or residual.stride(-1) != 1):
        return False
    if bias is not None and not (bias.dtype == torch.bfloat16 and bias.is_contiguous() and bias.is_cuda):
        return False
    # inputs that are not laid out for the kernel stay on the fallback, which they always took at these sizes
    for t in (a, b, out, residual):
        if t is not None and (t.stride(-1) != 1 or t.stride(0) % 8 or t.data_ptr() % 16):
            return False
    return out.dtype in (torch.bfloat16, torch.float32)


def gemm_reference(a, b, a_mn=False, b_mn=False, out=None, out_dtype=None, accumulate=False, alpha=1.0, bias=None):
    """fp32-accumulated PyTorch evaluation of the same contract (the oracle for the kernel)."""
    A = a.t() if a_mn else a
    B = b.t() if b_mn else b
    r = (A.float() @ B.float().t()) * alpha
    if bias is not None:
        r = r + bias.float()
    if out is not None:
        if accumulate:
            r = r + out.float()
        out.copy_(r.to(out.dtype))
        return out
    return r.to(out_dtype or a.dtype)


def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    a_mn: bool = False,
    b_mn: bool = False,
    out: Optional[torch.Tensor] = None,
    out_dtype: Optional[torch.dtype] = None,
    accumulate: bool = False,
    alpha: float = 1.0,
    bias: Optional[torch.Tensor] = None,
    tile_n: int = 0,
    max_ctas: int = 0,
    kernel: str = "auto",
    residual: Optional[torch.Tensor] = None,
    groups: Optional[dict] = None,
) -> torch.Tensor:
    """``out[M,N] (+)= alpha * A[M,K] @ B[N,K]^T (+ bias[N])``.

    ``a`` is stored ``[M,K]`` (or ``[K,M]`` when ``a_mn``), ``b`` is stored ``[N,K]`` (or ``[K,N]``
    when ``b_mn``). Inputs are bf16, accumulation is fp32, the output is bf16 or fp32.

    ``tile_n`` (CTA-pair kernel): 0 = by a rule on the sizes, 128 or 256 = tiles of that width, 512 = tiles of 256 columns
    with two pairs of CTAs each, half of the reduction a pair.

    ``groups`` (mixture-of-experts buffers, CTA-pair kernel only): ``{"counts": int32 device tensor,
    "m_rows": r}`` - rows of A come in groups of ``r`` slots (a multiple of 256) of which only the first
    ``counts[g]`` hold data and the rest is zero: tiles beyond the count are not computed, their output is
    zero. ``"k_rows": r`` - the same along the reduction dim (multiple of 64): empty k-blocks are skipped.
    ``"n_b": E, "bm_rows": R`` - ``b`` holds E stacked operands and rows ``[e*R, (e+1)*R)`` of A use the
    e-th (one launch for all local experts).
    """
    assert a.dim() == 2 and b.dim() == 2
    M, K = (a.shape[1], a.shape[0]) if a_mn else a.shape
    N, Kb = (b.shape[1], b.shape[0]) if b_mn else b.shape
    n_b = int(groups.get("n_b", 1)) if groups else 1
    if n_b > 1:                      # stacked B operands: [E*N, K] (or [E*K, N] when b_mn)
        if b_mn:
            Kb //= n_b
        else:
            N //= n_b
    assert K == Kb, f"reduction dims differ: {K} vs {Kb}"
    if out is None:
        out = torch.empty(M, N, dtype=out_dtype or torch.bfloat16, device=a.device)
        assert not accumulate
    if not _lib.use_kernels(a, b, out) or a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16 \
            or not _sizes_ok(a, b, M, N, K, a_mn, b_mn, out, groups, bias, residual):
        if n_b > 1:                  # reference: one product per stacked operand (inputs are zero beyond the counts)
            R = groups["bm_rows"]
            for e in range(n_b):
                be = b[e * K: (e + 1) * K] if b_mn else b[e * N: (e + 1) * N]
                gemm_reference(a[e * R: (e + 1) * R], be, a_mn, b_mn, out[e * R: (e + 1) * R], None, accumulate,
                               alpha, bias)
            return out
        r = gemm_reference(a, b, a_mn, b_mn, out, None, accumulate, alpha, bias)
        if residual is not None:
            r.add_(residual.to(r.dtype))
        return r
    if a.stride(-1) != 1:
        a = a.contiguous()
    if b.stride(-1) != 1:
        b = b.contiguous()
    assert out.stride(-1) == 1 and out.dtype in (torch.bfloat16, torch.float32)
    L = _lib.lib()
    use_pair = kernel == "2cta" or (kernel == "auto" and PAIR_KERNEL_DEFAULT and M >= 256 and N >= 256)
    pa, pb, po, fp32 = _pitch(a), _pitch(b), _pitch(out), int(out.dtype == torch.float32)
    pr = _pitch(residual) if residual is not None else 0
    head = (a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.addr(bias), M, N, K, pa, pb, po, int(a_mn), int(b_mn), fp32,
            int(accumulate), alpha, tile_n, max_ctas, _lib.addr(residual), pr)
    tail = (_lib.stream(), _lib.status_addr(a))
    if groups is not None:
        counts = groups.get("counts")
        assert counts is None or (counts.dtype == torch.int32 and counts.is_cuda)
        rc = L.atb_gemm_bf16_2cta_grouped(*head, _lib.addr(counts), int(groups.get("m_rows", 0)),
                                          int(groups.get("k_rows", 0)), (K if b_mn else N) if n_b > 1 else 0,
                                          int(groups.get("bm_rows", 0)), n_b, *tail)
        name = "atb_gemm_bf16_2cta_grouped"
    elif use_pair:
        rc = L.atb_gemm_bf16_2cta(*head, *tail)
        name = "atb_gemm_bf16_2cta"
    else:
        rc = L.atb_gemm_bf16(*head, *tail)
        name = "atb_gemm_bf16"
    if rc != 0:
        _lib.check(rc, f"{name} M={M} N={N} K={K}")
    return out


MAX_RAGGED_GROUPS = 64


def ragged_ok(x: torch.Tensor, w: torch.Tensor, b_mn: bool, n_groups: int) -> bool:
    """Whether ``gemm_ragged`` takes these operands: bf16 on the GPU, laid out for 16-byte loads and stores, and a
    reduction dim of whole 64-row blocks where the stacked operands follow each other along it."""
    N, K = (w.shape[2], w.shape[1]) if b_mn else (w.shape[1], w.shape[2])
    return (_lib.use_kernels(x, w) and _lib.lib().has("atb_gemm_bf16_2cta_ragged") and PAIR_KERNEL_DEFAULT
            and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and 0 < n_groups <= MAX_RAGGED_GROUPS
            and w.shape[0] == n_groups and x.dim() == 2 and x.shape[1] == K and N % 8 == 0
            and K % (64 if b_mn else 8) == 0 and w.is_contiguous() and x.stride(1) == 1 and x.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def gemm_ragged(x: torch.Tensor, w: torch.Tensor, sizes, b_mn: bool, gated: bool = False, keep_gate_up: bool = False):
    """Rows of ``x`` in consecutive groups of ``sizes`` rows (host numbers), group ``g`` times ``w[g]`` (``[K, N]``)
    when ``b_mn`` else times ``w[g]^T`` (``[N, K]``): one launch for all groups. See :func:`ragged_ok`.

    ``gated``: the weights hold gate | up features; returns ``(silu(gate) * up, gate | up)``, the second only with
    ``keep_gate_up`` (else None)."""
    M, K = x.shape
    N = w.shape[2] if b_mn else w.shape[1]
    N = N // 2 if gated else N
    out = torch.empty(M, N, dtype=x.dtype, device=x.device)
    gu = torch.empty(M, 2 * N, dtype=x.dtype, device=x.device) if gated and keep_gate_up else None
    rc = _lib.lib().atb_gemm_bf16_2cta_ragged(
        x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, _pitch(x), w.shape[2], N, int(b_mn),
        (ctypes.c_int * len(sizes))(*sizes), len(sizes), int(gated), _lib.addr(gu), _lib.stream(), _lib.status_addr(x))
    _lib.check(rc, f"atb_gemm_bf16_2cta_ragged M={M} N={N} K={K} groups={len(sizes)}")
    return (out, gu) if gated else out


def k_groups_ok(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor) -> bool:
    """Whether ``gemm_k_groups`` takes these operands: bf16 rows on the GPU in 16-byte pieces, stacked outputs."""
    return (_lib.use_kernels(a, b, out) and PAIR_KERNEL_DEFAULT and a.dim() == b.dim() == 2 and out.dim() == 3
            and a.dtype == b.dtype == torch.bfloat16 and out.dtype in (torch.bfloat16, torch.float32)
            and a.shape[0] == b.shape[0] > 0 and a.shape[1] % 8 == 0 and b.shape[1] % 8 == 0
            and tuple(out.shape[1:]) == (a.shape[1], b.shape[1]) and out.is_contiguous()
            and all(t.stride(1) == 1 and t.stride(0) % 8 == 0 for t in (a, b))
            and all(t.data_ptr() % 16 == 0 for t in (a, b, out)))


def gemm_k_groups(a: torch.Tensor, b: torch.Tensor, sizes, out: torch.Tensor, accumulate: bool) -> torch.Tensor:
    """``out[g] (+)= a_g^T b_g`` over consecutive groups of ``sizes`` rows (host numbers): one launch for up to 16 groups.
    See :func:`k_groups_ok`."""
    rc = _lib.lib().atb_gemm_bf16_2cta_kgroups(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), a.shape[1], b.shape[1], a.shape[0], a.stride(0), b.stride(0),
        (ctypes.c_int * len(sizes))(*sizes), len(sizes), int(out.dtype == torch.float32), int(accumulate), _lib.stream(),
        _lib.status_addr(a))
    _lib.check(rc, f"atb_gemm_bf16_2cta_kgroups T={a.shape[0]} M={a.shape[1]} N={b.shape[1]} groups={len(sizes)}")
    return out


def _linear_grads(ctx, dy2, x2, weight, need_dx, need_dw):
    """dx and dW of ``y = x W^T`` from ``dy``; dW goes straight into ``weight.main_grad`` when there is one."""
    dx = dw = None
    if need_dx:
        dx = gemm(dy2, weight, b_mn=True, out_dtype=x2.dtype).view(ctx.x_shape)
    if need_dw:
        mg = getattr(ctx.weight_ref, "main_grad", None)
        if mg is not None:
            first = getattr(ctx.weight_ref, "_atb_first", False)     # untouched buffer: overwrite, no zero fill
            gemm(dy2, x2, a_mn=True, b_mn=True, out=mg, accumulate=not first)
            ctx.weight_ref._atb_first = False
            ctx.weight_ref.grad_added_to_main_grad = True
        else:
            dw = gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=weight.dtype)
    return dx, dw


def gemm_swiglu(x2: torch.Tensor, weight: torch.Tensor, keep_gate_up: bool):
    """``act = silu(x Wg^T) * (x Wu^T)`` for the fused weight ``[Wg; Wu]`` in one kernel (gated epilogue of the
    CTA-pair GEMM); with ``keep_gate_up`` also the bf16 gate|up tensor ``[T, 2F]`` that the backward needs."""
    T, K = x2.shape
    F = weight.shape[0] // 2
    act = torch.empty(T, F, dtype=x2.dtype, device=x2.device)
    gu = torch.empty(T, 2 * F, dtype=x2.dtype, device=x2.device) if keep_gate_up else None
    rc = _lib.lib().atb_gemm_bf16_2cta_swiglu(
        x2.data_ptr(), weight.data_ptr(), act.data_ptr(), _lib.addr(gu), T, F, K, _pitch(x2), _pitch(weight), F, 2 * F,
        _lib.stream(), _lib.status_addr(x2))
    _lib.check(rc, f"atb_gemm_bf16_2cta_swiglu T={T} F={F} K={K}")
    return act, gu


class _LinearSwiGLU(torch.autograd.Function):
    """``swiglu(x @ W^T)`` with the activation computed in the GEMM epilogue. A pass that needs no gradient (the
    first pass of an activation-checkpointed block) never writes the ``[T, 2F]`` pre-activation; a pass that does
    writes it from the same epilogue, so the separate SwiGLU kernel and its read of that tensor disappear."""

    @staticmethod
    def forward(ctx, x, weight):
        shp = x.shape
        x2 = x.reshape(-1, shp[-1])
        x2 = x2 if x2.stride(-1) == 1 else x2.contiguous()
        need = ctx.needs_input_grad[0] or ctx.needs_input_grad[1]
        act, gu = gemm_swiglu(x2, weight, need)
        if need:
            ctx.save_for_backward(x2, weight, gu)
        ctx.x_shape, ctx.weight_ref = shp, weight
        return act.view(*shp[:-1], act.shape[-1])

    @staticmethod
    def backward(ctx, dact):
        from .elementwise import swiglu_backward

        x2, weight, gu = ctx.saved_tensors
        dgu = swiglu_backward(gu, dact.reshape(-1, dact.shape[-1]))
        dx, dw = _linear_grads(ctx, dgu, x2, weight, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        return dx, dw


def linear_swiglu(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``silu(x @ Wg.T) * (x @ Wu.T)`` for ``weight = [Wg; Wu]`` (``[2F, K]``), the gated MLP's first half."""
    from .elementwise import swiglu

    F = weight.shape[0] // 2
    if not (x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and _lib.use_kernels(x, weight)
            and _lib.lib().has("atb_gemm_bf16_2cta_swiglu") and F % 8 == 0 and x.shape[-1] % 8 == 0
            and weight.stride(-1) == 1 and PAIR_KERNEL_DEFAULT):
        return swiglu(linear(x, weight))
    return call(_LinearSwiGLU, x, weight)


class _LinearRope(torch.autograd.Function):
    """``rope(x @ W^T)`` with the rotation in the GEMM epilogue; its backward rotates the incoming gradient back in front of
    the projection's products."""

    @staticmethod
    def forward(ctx, x, weight, cos, sin, positions, nheads, head_dim, inplace_grad):
        shp = x.shape
        x2 = x.reshape(-1, shp[-1])
        x2 = x2 if x2.stride(-1) == 1 else x2.contiguous()
        T, K = x2.shape
        N = weight.shape[0]
        out = torch.empty(T, N, dtype=x2.dtype, device=x2.device)
        rc = _lib.lib().atb_gemm_bf16_2cta_rope(
            x2.data_ptr(), weight.data_ptr(), out.data_ptr(), T, N, K, _pitch(x2), _pitch(weight), N, cos.data_ptr(),
            sin.data_ptr(), _lib.addr(positions), cos.shape[0], nheads, head_dim, _lib.stream(), _lib.status_addr(x2))
        _lib.check(rc, f"atb_gemm_bf16_2cta_rope T={T} N={N} K={K}")
        ctx.save_for_backward(x2, weight, cos, sin, positions)
        ctx.x_shape, ctx.weight_ref, ctx.heads, ctx.inplace_grad = shp, weight, (nheads, head_dim), inplace_grad
        return out.view(*shp[:-1], N)

    @staticmethod
    def backward(ctx, dy):
        from .elementwise import _rope_launch

        x2, weight, cos, sin, positions = ctx.saved_tensors
        own = ctx.inplace_grad or not dy.is_contiguous()        # a gradient, or a copy of it, to write into
        src = dy.contiguous().view(-1, dy.shape[-1])
        dst = src if own else torch.empty_like(src)
        _rope_launch(dst, src, cos, sin, positions, *ctx.heads, True)
        dx, dw = _linear_grads(ctx, dst, x2, weight, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        return dx, dw, None, None, None, None, None, None


def linear_rope(x: torch.Tensor, weight: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, nheads: int, head_dim: int,
                positions: Optional[torch.Tensor] = None, inplace_grad: bool = False) -> torch.Tensor:
    """``rope(linear(x, weight), cos, sin, nheads, head_dim, positions)`` in one kernel where the pair kernel runs (from 256
    tokens on) and whole 128-column halves of its tiles are rotated or not.

    ``inplace_grad``: the backward pass overwrites the incoming gradient instead of writing a new tensor; only where that
    gradient is a temporary, as it is when the result goes straight into attention."""
    from .elementwise import rope

    T = x.numel() // max(x.shape[-1], 1)
    if not (x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and _lib.use_kernels(x, weight, cos, sin, positions)
            and PAIR_KERNEL_DEFAULT and T >= 256 and head_dim in (64, 128) and weight.dim() == 2
            and weight.shape[1] == x.shape[-1] and weight.shape[0] % 128 == 0
            and (nheads * head_dim) % 128 == 0 and 0 < nheads * head_dim <= weight.shape[0] and x.shape[-1] % 8 == 0
            and weight.stride(-1) == 1 and weight.stride(0) % 8 == 0 and weight.data_ptr() % 16 == 0
            and x.data_ptr() % 16 == 0 and (x.dim() < 2 or x.is_contiguous()) and cos.dtype == torch.float32
            and sin.dtype == torch.float32 and cos.is_contiguous() and sin.is_contiguous()
            and cos.shape == sin.shape and cos.dim() == 2 and cos.shape[1] == head_dim // 2
            and cos.data_ptr() % 16 == 0 and sin.data_ptr() % 16 == 0
            and (positions is None or (positions.numel() == T and positions.is_contiguous()))):
        return rope(linear(x, weight), cos, sin, nheads, head_dim, positions, inplace=inplace_grad)
    if positions is not None and positions.dtype != torch.int32:
        positions = positions.to(torch.int32)
    return call(_LinearRope, x, weight, cos, sin, positions, nheads, head_dim, inplace_grad)


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, residual):
        shp = x.shape
        x2 = x.reshape(-1, shp[-1])
        ctx.save_for_backward(x2, weight)
        ctx.has_bias = bias is not None
        ctx.has_res = residual is not None
        ctx.x_shape = shp
        ctx.weight_ref = weight
        if residual is not None:
            # out = residual + x W^T : the epilogue reads the residual stream and adds it before the store
            r2 = residual.reshape(-1, weight.shape[0])
            r2 = r2 if r2.stride(-1) == 1 else r2.contiguous()
            out = gemm(x2, weight, bias=bias, out_dtype=x.dtype, residual=r2)
        else:
            out = gemm(x2, weight, bias=bias, out_dtype=x.dtype)
        return out.view(*shp[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, weight = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if dy2.stride(-1) != 1:
            dy2 = dy2.contiguous()
        db = dres = None
        dx, dw = _linear_grads(ctx, dy2, x2, weight, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy2.sum(0)
        if ctx.has_res and ctx.needs_input_grad[3]:
            dres = dy
        return dx, dw, db, dres


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
           residual: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``residual + x @ weight.T + bias`` with the tcgen05 GEMM in forward, dgrad and wgrad."""
    if x.dtype != torch.bfloat16 or not _lib.use_kernels(x, weight):
        y = torch.nn.functional.linear(x, weight.to(x.dtype), None if bias is None else bias.to(x.dtype))
        return y if residual is None else residual + y
    return call(_Linear, x, weight, bias, residual)
