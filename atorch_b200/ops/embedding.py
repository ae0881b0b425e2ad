"""Token embedding whose gradient goes straight into ``weight.main_grad`` (``csrc/embedding.cu``)."""
from __future__ import annotations

import ctypes
import functools

import torch
import torch.nn as nn
from torch.nn.modules import module as nn_module
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

from .. import _lib
from .function import watched


@functools.cache
def _words():
    fn = _lib.lib().atb_embedding_bwd_scratch
    fn.restype = ctypes.c_longlong
    return fn


def embedding_grad(dy: torch.Tensor, ids: torch.Tensor, out: torch.Tensor, accumulate: bool) -> torch.Tensor:
    """``out[v] (+)= sum of dy over the tokens whose id is v`` (bf16 ``dy``; fp32 sums in an order that the ids alone decide)."""
    V, H = out.shape
    T = ids.numel()
    dy = dy.reshape(T, H).contiguous()
    if dy.data_ptr() % 16:
        dy = dy.clone()
    ids = ids.contiguous()
    scratch = torch.empty(_words()(T, V, H), dtype=torch.int32, device=out.device)
    rc = _lib.lib().atb_embedding_bwd(dy.data_ptr(), ids.data_ptr(), out.data_ptr(), scratch.data_ptr(), T, V, H,
                                      int(out.dtype == torch.float32), int(accumulate), _lib.stream())
    _lib.check(rc, f"atb_embedding_bwd T={T} V={V} H={H}")
    return out


class _EmbeddingFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, weight):
        ctx.save_for_backward(ids)
        ctx.weight_ref = weight
        ctx.weight_shape = weight.shape
        return torch.embedding(weight, ids)

    @staticmethod
    def backward(ctx, dy):
        ids, = ctx.saved_tensors
        if torch.is_grad_enabled() or watched(dy, ids):   # a second derivative, a batch of gradients, a dispatch mode
            return None, torch.ops.aten.embedding_dense_backward(dy, ids, ctx.weight_shape[0], -1, False)
        mg = getattr(ctx.weight_ref, "main_grad", None)
        if mg is None:
            return None, embedding_grad(dy, ids, torch.empty(ctx.weight_shape, dtype=dy.dtype, device=dy.device), False)
        first = getattr(ctx.weight_ref, "_atb_first", False)         # untouched buffer: every row is written
        if mg.dtype in (torch.bfloat16, torch.float32) and mg.is_contiguous() and mg.data_ptr() % 16 == 0:
            embedding_grad(dy, ids, mg, not first)
        else:
            dw = embedding_grad(dy, ids, torch.empty(ctx.weight_shape, dtype=dy.dtype, device=dy.device), False)
            mg.copy_(dw) if first else mg.add_(dw)
        ctx.weight_ref._atb_first = False
        ctx.weight_ref.grad_added_to_main_grad = True
        return None, None


def _plain(m: nn.Module) -> bool:
    """Nothing but ``F.embedding`` on the weight: no option of it, and nobody who watches or replaces the call."""
    return (type(m) is nn.Embedding and m.padding_idx is None and m.max_norm is None and not m.sparse
            and not m.scale_grad_by_freq and "forward" not in m.__dict__ and m._compiled_call_impl is None
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks)
            and not nn_module._has_any_global_hook()
            and all(type(mode) is DeviceContext for mode in _get_current_function_mode_stack()))


def embedding(module: nn.Module, ids: torch.Tensor) -> torch.Tensor:
    """``module(ids)``; a plain bf16 ``nn.Embedding`` on the GPU that trains takes its gradient from the kernels."""
    if type(ids) is torch.Tensor and ids.is_cuda and ids.dtype == torch.int64 and torch.is_grad_enabled() and _plain(module):
        w = module.weight
        if (w.requires_grad and type(w) is nn.Parameter and w.is_cuda and w.dtype == torch.bfloat16 and w.shape[1] % 8 == 0
                and ids.numel() < 2 ** 30 and w.numel() > 0 and not w._backward_hooks and not w._post_accumulate_grad_hooks
                and _lib.use_kernels(w) and not watched(ids, w)):
            return _EmbeddingFn.apply(ids, w)
    return module(ids)
