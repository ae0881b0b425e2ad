"""The embedding's autograd function serves whoever the library's gradient serves (csrc/embedding.cu is for the rest)."""
import pytest
import torch
import torch.nn.functional as F
from torch.utils._python_dispatch import TorchDispatchMode

from atorch_b200.ops.embedding import _EmbeddingFn


class _Seen(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names = getattr(self, "names", []) + [func.overloadpacket.__name__]
        return func(*args, **(kwargs or {}))


def _second(apply):
    w = (torch.arange(60.0).view(10, 6) / 7).requires_grad_()
    x = apply(torch.tensor([3, 3, 1, 9]), w)
    (g,) = torch.autograd.grad((x ** 3).sum(), w, create_graph=True)
    return torch.autograd.grad((g ** 2).sum(), w, create_graph=True)[0].detach()


def _batch(apply):
    w = torch.ones(10, 6, requires_grad=True)
    w.main_grad = torch.zeros(10, 6)
    x = apply(torch.tensor([[3, 3], [1, 9]]), w)
    return torch.autograd.grad(x, w, torch.arange(72.0).view(3, 2, 2, 6), is_grads_batched=True)[0]


def _mode(apply):
    w = torch.ones(10, 6, requires_grad=True)
    x = apply(torch.tensor([3, 3, 1]), w)
    with _Seen() as seen:
        (g,) = torch.autograd.grad((x * 2).sum(), w)
    assert "embedding_dense_backward" in seen.names
    return g


@pytest.mark.parametrize("use", [_second, _batch, _mode])
def test_gradients_of_gradients_batches_and_modes(use):
    assert torch.equal(use(_EmbeddingFn.apply), use(lambda ids, w: F.embedding(ids, w)))
