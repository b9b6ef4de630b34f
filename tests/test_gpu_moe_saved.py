"""The expert layer's backward on tensors that a saved-tensor hook has moved."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _grads(unpack, python, monkeypatch):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops import kernels

    if python:
        monkeypatch.setattr(kernels, "traced_or_dual", lambda *t: True)
    g = torch.Generator(device="cuda").manual_seed(2)
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(torch.bfloat16)
    x, w13, w2, dy = mk(90, 128), mk(8, 144, 128, scale=0.1), mk(8, 128, 72, scale=0.1), mk(90, 128)
    gate, idx = torch.rand(90, 2, device="cuda", generator=g), torch.rand(90, 8, device="cuda", generator=g).topk(2, 1).indices
    leaves = [t.requires_grad_() for t in (x, gate, w13, w2)]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = OF.local_moe(x, gate, idx, w13, w2)
    y.backward(dy)
    return [t.grad for t in leaves]


def _off_the_boundary(t):
    return torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)[1:].view(t.shape).copy_(t)


def _strided(t):
    return torch.empty(*t.shape, 2, device=t.device, dtype=t.dtype)[..., 0].copy_(t)


@pytest.mark.parametrize("python", [False, True])
@pytest.mark.parametrize("unpack", [_off_the_boundary, _strided])
def test_moved_tensors_give_the_same_gradients(unpack, python, monkeypatch):
    want = _grads(lambda t: t, python, monkeypatch)
    for a, b in zip(_grads(unpack, python, monkeypatch), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("shape", [(8, 144, 128), (8, 128, 72), (90, 2)])  # w13, w2, gate weights
@pytest.mark.parametrize("change", [lambda t: t.cpu(), lambda t: t.double(), lambda t: t[:, :1]])
def test_what_the_kernels_cannot_read_is_refused(shape, change, monkeypatch):
    with pytest.raises(RuntimeError, match="saved tensors|another layer call|bad dy"):
        _grads(lambda t: change(t) if t.shape == shape and t.is_floating_point() else t, False, monkeypatch)
