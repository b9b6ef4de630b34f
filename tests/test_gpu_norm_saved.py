"""RMSNorm's backward on what the graph hands back: a weight that a saved-tensor hook has moved."""

import pytest
import torch

pytestmark = pytest.mark.gpu

H = 1032


def _grads(monkeypatch, python, unpack=None):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops import kernels

    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    x, d, w, dy = mk(33, H).requires_grad_(), mk(33, H).requires_grad_(), mk(H).requires_grad_(), mk(33, H)
    with monkeypatch.context() as m:
        if python:
            m.setattr(kernels, "traced_or_dual", lambda *t: True)
        with torch.autograd.graph.saved_tensors_hooks(
                lambda t: t, lambda t: unpack(t) if unpack and t.shape == w.shape and t.dtype == w.dtype else t):
            y = OF.add_rmsnorm(x, d, w)[1]
        y.backward(dy)
    return x.grad, d.grad, w.grad


def _off_the_boundary(t):
    return torch.empty(H + 1, device="cuda", dtype=t.dtype)[1:].copy_(t)


def _strided(t):
    return torch.empty(2 * H, device="cuda", dtype=t.dtype)[::2].copy_(t)


@pytest.mark.parametrize("python", [False, True])
@pytest.mark.parametrize("unpack", [_off_the_boundary, _strided])
def test_a_moved_weight_gives_the_same_gradients(python, unpack, monkeypatch):
    want = _grads(monkeypatch, python)
    for a, b in zip(_grads(monkeypatch, python, unpack), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("python", [False, True])
@pytest.mark.parametrize("unpack", [lambda t: t.cpu(), lambda t: t.float(), lambda t: t[:8]])
def test_a_weight_that_the_kernel_cannot_read_is_refused(python, unpack, monkeypatch):
    with pytest.raises(RuntimeError, match="add_rmsnorm_grad"):
        _grads(monkeypatch, python, unpack)


@pytest.mark.parametrize("python", [False, True])
@pytest.mark.parametrize("shape", [(1, H), (H, 1)])
def test_a_weight_of_more_dimensions_gets_a_gradient_of_its_shape(python, shape, monkeypatch):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops import kernels

    if python:
        monkeypatch.setattr(kernels, "traced_or_dual", lambda *t: True)
    x = torch.randn(5, H, device="cuda").to(torch.bfloat16)
    flat = torch.randn(H, device="cuda").to(torch.bfloat16).requires_grad_()
    w = flat.detach().clone().view(shape).requires_grad_()
    for weight in (flat, w):
        OF.rmsnorm(x, weight).float().pow(2).sum().backward()
    assert torch.equal(w.grad, flat.grad.view(shape))
