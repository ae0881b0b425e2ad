"""Who looks at the operators' calls, and calls of their autograd functions where nothing can ask for a gradient."""
from __future__ import annotations

from typing import Optional

import torch
from torch.autograd import forward_ad


def watched(*ts: Optional[torch.Tensor]) -> bool:
    """Whether something other than reverse-mode autograd looks at operations on these tensors (a functorch transform,
    forward-mode differentiation, a batch of gradients, a tracer or another dispatch mode, a tensor subclass): kernels called by
    address would hide them from it, tensor operations do not."""
    return (torch._C._functorch.peek_interpreter_stack() is not None or torch.jit.is_tracing()
            or torch.compiler.is_compiling() or torch._C._len_torch_dispatch_stack() > 0
            or torch._ops._len_torch_dispatch_stack_pre_dispatch() > 0
            or any(type(t) not in (torch.Tensor, torch.nn.Parameter) or torch._C._functorch.is_legacy_batchedtensor(t)
                   or forward_ad.unpack_dual(t).tangent is not None for t in ts if t is not None))


class _NoGradContext:
    """What ``forward`` finds in place of its autograd context: no input needs a gradient, nothing is kept."""

    needs_input_grad = (False,) * 16

    def save_for_backward(self, *tensors):
        pass


def call(function, *args):
    """``function.apply(*args)``; where gradients are switched off, its ``forward`` alone. ``apply`` builds a node, unpacks
    and re-wraps every argument and reports ``needs_input_grad`` by the flags of the inputs even then (5 of the 21 us that a
    linear layer takes on the host, and the gate|up tensor of the first pass of a checkpointed block was written for nobody:
    90 MB per layer at 4096 x 5504). Anything that looks into calls, a transform, forward-mode differentiation or a tracer,
    still gets ``apply``, which either serves it or refuses. (Under a dispatch mode and for a tensor subclass ``apply`` runs the
    same ``forward`` on the same arguments.) A tensor that has outlived its transform has no address, which ``forward`` asks for
    before it launches anything; ``apply`` unwraps it (unwrapping every argument here took 0.5 us a call)."""
    if torch.is_grad_enabled() or torch._C._are_functorch_transforms_active() or forward_ad._current_level >= 0 \
            or torch._C._get_tracing_state() is not None:
        return function.apply(*args)
    try:
        return function.forward(_NoGradContext(), *args)
    except RuntimeError:
        if not any(type(a) is torch.Tensor and torch._C._functorch.is_functorch_wrapped_tensor(a) for a in args):
            raise
    return function.apply(*args)
