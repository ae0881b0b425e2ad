"""Token permutation for mixture-of-experts and the grouped GEMM that consumes it.

``permute(tokens, expert_idx)``: stable sort of the flattened ``[T, k]`` expert ids; row j of the result
is token ``sorted[j] // k``. ``unpermute`` scatters expert outputs back, weights them with the routing
probabilities and sums over the k choices. Counts per expert stay on the device
(``tokens_per_expert``), the host only learns them when a variable-size exchange needs split lists.

``grouped_gemm(x, w, batch_sizes, trans_b)``: consecutive row groups of ``x`` times one weight per
group, each product on the tcgen05 GEMM (``ops.gemm``) with its forward / dgrad / wgrad layouts.
(Reference semantics: atorch/modules/moe/token_dispatcher.py:89-161; grouped_gemm.ops.gmm used at
atorch/modules/moe/grouped_gemm_moe.py:841-850; megablocks sort/histogram ops at :566-596.)
"""
from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import torch

from .. import _lib
from .elementwise import swiglu, swiglu_backward
from .function import watched
from .gemm import gemm, gemm_k_groups, gemm_ragged, k_groups_ok, linear, ragged_ok


def tokens_per_expert(expert_idx: torch.Tensor, num_experts: int) -> torch.Tensor:
    """int64 histogram ``[num_experts]`` of the routed expert ids (device resident, deterministic)."""
    return torch.bincount(expert_idx.reshape(-1), minlength=num_experts)


def _rows_ok(rows: torch.Tensor, order: torch.Tensor) -> bool:
    """Whether the row kernels (csrc/moe_local.cu) take these rows: bf16 on the GPU in 16-byte pieces, int64 order."""
    return (_lib.use_kernels(rows, order) and rows.dtype == torch.bfloat16 and rows.dim() == 2 and rows.shape[1] % 8 == 0
            and rows.shape[1] > 0 and order.dtype == torch.int64 and order.dim() == 1 and order.is_contiguous()
            and 0 < order.numel() < 1 << 31 and not watched(rows, order))


def _slots(order: torch.Tensor) -> torch.Tensor:
    """Row of the sorted buffer of every (token, choice)."""
    slot = torch.empty(order.numel(), dtype=torch.int32, device=order.device)
    _lib.check(_lib.lib().atb_invert_perm(order.data_ptr(), slot.data_ptr(), order.numel(), _lib.stream()), "atb_invert_perm")
    return slot


def _gather_sum(rows, slot, w, T, k):
    out = torch.empty(T, rows.shape[1], dtype=rows.dtype, device=rows.device)
    rc = _lib.lib().atb_moe_gather_sum(rows.data_ptr(), slot.data_ptr(), _lib.addr(w), 0 if w is None else _lib.DT[w.dtype],
                                       out.data_ptr(), T, k, rows.shape[1], _lib.stream())
    _lib.check(rc, "atb_moe_gather_sum")
    return out


def _packed(t: torch.Tensor) -> torch.Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


class _Permute(torch.autograd.Function):
    """Keeps the inverse of ``order`` for its backward pass, not ``order``, which is the caller's."""

    @staticmethod
    def forward(ctx, tokens, order, k, slot):
        ctx.k, ctx.T = k, tokens.shape[0]
        if slot is None:
            ctx.save_for_backward(_slots(order) if ctx.needs_input_grad[0] else None)
            return tokens.index_select(0, order // k)
        ctx.save_for_backward(slot)
        src = _packed(tokens)                   # ids sorted by route(): their places are rows for certain
        out = torch.empty(order.numel(), src.shape[1], dtype=src.dtype, device=src.device)
        rc = _lib.lib().atb_moe_gather_rows(src.data_ptr(), order.data_ptr(), out.data_ptr(), order.numel(), k, src.shape[1],
                                            _lib.stream())
        _lib.check(rc, "atb_moe_gather_rows")
        return out

    @staticmethod
    def backward(ctx, dy):
        (slot,) = ctx.saved_tensors
        if torch.is_grad_enabled() or watched(dy):     # operations that autograd and the others can follow
            return dy.index_select(0, slot).view(ctx.T, ctx.k, -1).sum(1), None, None, None
        return _gather_sum(_packed(dy), slot, None, ctx.T, ctx.k), None, None, None


class _Unpermute(torch.autograd.Function):
    @staticmethod
    def forward(ctx, rows, order, probs, k, slot):
        # the rows are read again only for the gradient of the probabilities
        ctx.save_for_backward(rows if ctx.needs_input_grad[2] else None, order, probs)
        ctx.k, ctx.sorted = k, slot is not None
        slot = _slots(order) if slot is None else slot
        return _gather_sum(_packed(rows), slot, None if probs is None else probs.contiguous(), order.numel() // k, k)

    @staticmethod
    def backward(ctx, dout):
        rows, order, probs = ctx.saved_tensors
        need_dw = ctx.needs_input_grad[2]
        if torch.is_grad_enabled() or watched(dout):   # operations that autograd and the others can follow
            d, dw = dout.index_select(0, order // ctx.k), None
            if need_dw:
                dots = (rows * d).sum(-1).to(probs.dtype)
                dw = torch.zeros_like(dots).index_copy(0, order, dots).view(probs.shape)
            if probs is not None:
                d = d * probs.reshape(-1, 1).index_select(0, order).to(d.dtype)
            return d, None, dw, None, None
        w, dout = None if probs is None else probs.contiguous(), _packed(dout)
        rows = _packed(rows) if need_dw else None
        n, H = order.numel(), dout.shape[1]
        drows = torch.empty(n, H, dtype=dout.dtype, device=dout.device) if ctx.needs_input_grad[0] else None
        # an order of the caller's own may leave a choice out
        dw = (torch.empty_like if ctx.sorted else torch.zeros_like)(w) if need_dw else None
        rc = _lib.lib().atb_moe_ungather(dout.data_ptr(), _lib.addr(rows), order.data_ptr(), _lib.addr(w),
                                         2 if w is None else _lib.DT[w.dtype], _lib.addr(drows), _lib.addr(dw), n, ctx.k, H,
                                         _lib.stream())
        _lib.check(rc, "atb_moe_ungather")
        return drows, None, None if dw is None else dw.view(probs.shape), None, None


def permute(tokens: torch.Tensor, expert_idx: torch.Tensor, num_out_tokens: Optional[int] = None
            ) -> Tuple[torch.Tensor, torch.Tensor]:
    """tokens ``[T, H]``, expert_idx ``[T, k]`` (or ``[T]``) -> (permuted ``[T*k, H]``, sorted_indices)."""
    k = expert_idx.shape[1] if expert_idx.dim() > 1 else 1
    flat = expert_idx.reshape(-1)
    sorted_idx = torch.argsort(flat, stable=True)
    if num_out_tokens is None and _rows_ok(tokens, sorted_idx) and sorted_idx.numel() == tokens.shape[0] * k:
        return _Permute.apply(tokens, sorted_idx, k, None), sorted_idx
    if num_out_tokens is not None:
        sorted_idx = sorted_idx[:num_out_tokens]
    return tokens.index_select(0, sorted_idx // k), sorted_idx


# One block sorts up to 32768 ids of up to 256 experts no slower than the radix sort (see csrc/moe_local.cu); with the launches
# and the histogram's synchronisation counted it is 53 us against 215 for 8192 ids, 127 against 215 for 32768 of 256 experts.
ROUTE_MAX_IDS, ROUTE_MAX_EXPERTS = 32768, 256


def route(tokens: torch.Tensor, expert_idx: torch.Tensor, num_experts: int):
    """``(tokens_per_expert(expert_idx, num_experts), *permute(tokens, expert_idx), slots)`` from one kernel that counts and
    sorts and one that gathers. ``slots`` (None on the general path) is for :func:`unpermute`. Ids outside
    ``[0, num_experts)`` are not counted: the group sizes then no longer cover the rows, which the grouped GEMMs and the
    exchange refuse."""
    k = expert_idx.shape[1] if expert_idx.dim() > 1 else 1
    flat = expert_idx.reshape(-1)
    if not (_rows_ok(tokens, flat) and flat.numel() == tokens.shape[0] * k and flat.numel() <= ROUTE_MAX_IDS
            and 0 < num_experts <= ROUTE_MAX_EXPERTS):
        return (tokens_per_expert(expert_idx, num_experts), *permute(tokens, expert_idx), None)
    # the caller's own: changing the counts in place must not touch `order`, which unpermute() keeps for its backward pass
    counts = torch.empty(num_experts, dtype=torch.int64, device=flat.device)
    order = torch.empty(flat.numel(), dtype=torch.int64, device=flat.device)
    slot = torch.empty(flat.numel(), dtype=torch.int32, device=flat.device)
    rc = _lib.lib().atb_moe_sort_ids(flat.data_ptr(), flat.numel(), num_experts, counts.data_ptr(), order.data_ptr(),
                                  slot.data_ptr(), _lib.stream())
    _lib.check(rc, "atb_moe_sort_ids")
    return counts, _Permute.apply(tokens, order, k, slot), order, slot


def unpermute(permuted: torch.Tensor, sorted_idx: torch.Tensor, probs: Optional[torch.Tensor] = None,
              topk: int = 1, num_tokens: Optional[int] = None, slots: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Inverse of :func:`permute`: ``[T*k, H] -> [T, H]`` with optional prob-weighted sum over k. ``slots``: the inverse
    of ``sorted_idx`` where :func:`route` made it (computed here otherwise)."""
    n_slots = (num_tokens * topk) if num_tokens is not None else (probs.numel() if probs is not None
                                                                   else sorted_idx.numel())
    if topk >= 1 and _rows_ok(permuted, sorted_idx) and n_slots == sorted_idx.numel() == permuted.shape[0] \
            and n_slots % topk == 0 and (probs is None or (probs.numel() == n_slots and probs.is_cuda
                                                           and probs.dtype in (torch.bfloat16, torch.float32)
                                                           and not watched(probs))):
        return _Unpermute.apply(permuted, sorted_idx, probs, topk, slots)
    return unpermute_reference(permuted, sorted_idx, probs, topk, n_slots)


def unpermute_reference(permuted, sorted_idx, probs, topk, n_slots):
    out = torch.zeros(n_slots, permuted.shape[-1], dtype=permuted.dtype, device=permuted.device)
    out = out.index_copy(0, sorted_idx, permuted)
    out = out.view(-1, topk, permuted.shape[-1])
    if probs is not None:
        out = out * probs.view(-1, topk, 1).to(out.dtype)
    return out.sum(dim=1)


class _GroupedLinear(torch.autograd.Function):
    """y[g] = x[g] @ W[g]^T for consecutive row groups (W stored [G, N, K]), or x[g] @ W[g] (W stored [G, K, N])
    when ``b_mn``: the GEMM reads either as it lies in memory. Forward, dgrad and wgrad are one launch each over all
    groups (wgrad: up to 16) where the kernel takes the operands."""

    @staticmethod
    def _rows(x, w, sizes, b_mn):
        if ragged_ok(x, w, b_mn, len(sizes)):
            return gemm_ragged(x, w, sizes, b_mn)
        out = torch.empty(x.shape[0], w.shape[2] if b_mn else w.shape[1], dtype=x.dtype, device=x.device)
        r = 0
        for g, n in enumerate(sizes):
            if n:
                gemm(x[r: r + n], w[g], b_mn=b_mn, out=out[r: r + n])
            r += n
        return out

    @staticmethod
    def forward(ctx, x, w, sizes: Tuple[int, ...], b_mn: bool):
        ctx.sizes, ctx.b_mn = sizes, b_mn
        ctx.save_for_backward(x, w)
        return _GroupedLinear._rows(x, w, sizes, b_mn)

    @staticmethod
    def _grads(x, w, dy, sizes, b_mn, need_dx, need_dw):
        dx = _GroupedLinear._rows(dy, w, sizes, not b_mn).to(x.dtype) if need_dx else None
        if not need_dw:
            return dx, None
        mg = getattr(w, "main_grad", None)
        dw = mg if mg is not None else torch.empty(w.shape, dtype=w.dtype, device=w.device)
        a, b = (x, dy) if b_mn else (dy, x)             # dW[g] = a[g]^T b[g]
        if len(sizes) == dw.shape[0] and k_groups_ok(a, b, dw):
            gemm_k_groups(a, b, sizes, dw, mg is not None)      # writes every group
        else:
            if mg is None:
                dw.zero_()                              # groups without rows, and weights that have no group
            r = 0
            for g, n in enumerate(sizes):
                if n:
                    gemm(a[r: r + n], b[r: r + n], a_mn=True, b_mn=True, out=dw[g], accumulate=mg is not None)
                r += n
        if mg is not None:
            w.grad_added_to_main_grad = True
            return dx, None
        return dx, dw

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        return (*_GroupedLinear._grads(x, w, dy.contiguous(), ctx.sizes, ctx.b_mn, *ctx.needs_input_grad[:2]), None, None)


class _GroupedSwiGLU(torch.autograd.Function):
    """``swiglu`` of :class:`_GroupedLinear` with the activation in the epilogue of its one launch. The gate | up rows
    are written only when there is a gradient to come."""

    @staticmethod
    def forward(ctx, x, w, sizes: Tuple[int, ...], b_mn: bool):
        need = ctx.needs_input_grad[0] or ctx.needs_input_grad[1]
        act, gu = gemm_ragged(x, w, sizes, b_mn, gated=True, keep_gate_up=need)
        if need:
            ctx.save_for_backward(x, w, gu)
        ctx.sizes, ctx.b_mn = sizes, b_mn
        return act

    @staticmethod
    def backward(ctx, dact):
        x, w, gu = ctx.saved_tensors
        return (*_GroupedLinear._grads(x, w, swiglu_backward(gu, dact), ctx.sizes, ctx.b_mn, *ctx.needs_input_grad[:2]),
                None, None)


def grouped_gemm(a: torch.Tensor, b: torch.Tensor, batch_sizes, trans_b: bool = False) -> torch.Tensor:
    """``gmm``: rows of ``a`` are split by ``batch_sizes`` (CPU ints / tensor); group g is multiplied by
    ``b[g]`` (``[K, N]``) or ``b[g]^T`` when ``trans_b`` (``[N, K]``)."""
    sizes = tuple(int(s) for s in (batch_sizes.tolist() if isinstance(batch_sizes, torch.Tensor) else batch_sizes))
    assert sum(sizes) == a.shape[0], "batch_sizes must cover all rows"
    return _GroupedLinear.apply(a, b, sizes, not trans_b)


def grouped_gemm_swiglu(a: torch.Tensor, b: torch.Tensor, batch_sizes, trans_b: bool = False) -> torch.Tensor:
    """``swiglu(grouped_gemm(a, b, batch_sizes, trans_b))`` for weights of gate | up features, in one kernel where the
    ragged launch takes the operands and the features come in 16-byte pieces (which the separate kernel needs too)."""
    N = b.shape[-2] if trans_b else b.shape[-1]
    if a.dim() == 2 and b.dim() == 3 and N % 16 == 0 and ragged_ok(a, b, not trans_b, b.shape[0]):
        sizes = tuple(int(s) for s in (batch_sizes.tolist() if isinstance(batch_sizes, torch.Tensor) else batch_sizes))
        assert sum(sizes) == a.shape[0], "batch_sizes must cover all rows"
        if len(sizes) == b.shape[0]:
            return _GroupedSwiGLU.apply(a, b, sizes, not trans_b)
        batch_sizes = sizes
    return swiglu(grouped_gemm(a, b, batch_sizes, trans_b))
