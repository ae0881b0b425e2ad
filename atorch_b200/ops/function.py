"""Calls of the operators' autograd functions where nothing can ask for a gradient."""
from __future__ import annotations

import torch
from torch.autograd import forward_ad


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
    still gets ``apply``, which either serves it or refuses."""
    if torch.is_grad_enabled() or torch._C._are_functorch_transforms_active() or forward_ad._current_level >= 0 \
            or torch._C._get_tracing_state() is not None:
        return function.apply(*args)
    return function.forward(_NoGradContext(), *args)
