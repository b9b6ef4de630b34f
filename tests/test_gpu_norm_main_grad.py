"""The gradient of a norm's weight under the fused optimizer: added to ``main_grad`` where nothing else waits for it, and
autograd's as of any parameter where something does."""

import pytest
import torch

pytestmark = pytest.mark.gpu

H = 264


@pytest.fixture(params=[False, True], ids=["native", "python"])
def norm(request, monkeypatch):
    """(x, weight, run) of one norm; ``run`` makes its forward and leaves the result's gradient bound."""
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops import kernels

    if request.param:
        monkeypatch.setattr(kernels, "traced_or_dual", lambda *t: True)
    g = torch.Generator(device="cuda").manual_seed(7)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    x, w, dy = mk(65, H).requires_grad_(), mk(H).requires_grad_(), mk(65, H)
    return x, w, lambda: (OF.rmsnorm(x, w).float() * dy.float()).sum()


def _plain_grad(norm):
    x, w, run = norm
    return torch.autograd.grad(run(), w)[0]


def _tensor_hook(w, seen):
    w.register_hook(lambda g: seen.append(g.clone()))


def _post_accumulate_hook(w, seen):
    w.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))


def _accumulator_hook(w, seen):
    node = w.view_as(w).grad_fn.next_functions[0][0]
    node.register_hook(lambda gi, go: seen.append(go[0].clone()))
    return node  # (the weight does not keep it)


def _accumulator_prehook(w, seen):
    node = w.view_as(w).grad_fn.next_functions[0][0]
    node.register_prehook(lambda go: seen.append(go[0].clone()))
    return node


def test_unwatched_gradients_go_to_the_buffer(norm):
    x, w, run = norm
    want = _plain_grad(norm)
    w.main_grad = torch.full((H,), 0.5, device="cuda")
    run().backward()
    assert w.grad is None
    # the fp32 sum that the other form rounds to bf16, added to 0.5 in fp32
    assert torch.allclose(w.main_grad - 0.5, want.float(), rtol=2.0 ** -8, atol=2.0 ** -20)


@pytest.mark.parametrize("watch", [_tensor_hook, _post_accumulate_hook, _accumulator_hook, _accumulator_prehook])
def test_hooks_of_the_weight_run(norm, watch):
    x, w, run = norm
    want = _plain_grad(norm)
    w.main_grad = torch.zeros(H, device="cuda")
    seen = []
    keep = watch(w, seen)
    run().backward()
    assert len(seen) == 1 and torch.equal(seen[0], want) and torch.equal(w.grad, want) and not w.main_grad.any()
    del keep


def test_gradients_that_are_asked_for_are_returned(norm):
    x, w, run = norm
    want = _plain_grad(norm)
    w.main_grad = torch.zeros(H, device="cuda")
    assert torch.equal(torch.autograd.grad(run(), w)[0], want)
    run().backward(inputs=[w])
    assert torch.equal(w.grad, want) and not w.main_grad.any()
    w.grad = None
    assert torch.autograd.grad(run(), x)[0].shape == x.shape
    assert w.grad is None and not w.main_grad.any()


@pytest.mark.parametrize("buffer", [
    lambda: torch.zeros(H, device="cuda", dtype=torch.bfloat16),
    lambda: torch.zeros(2 * H, device="cuda")[::2],
    lambda: torch.zeros(H),
])
def test_buffers_that_the_kernel_cannot_add_to(norm, buffer):
    x, w, run = norm
    want = _plain_grad(norm)
    w.main_grad = buffer()
    run().backward()
    assert torch.equal(w.grad, want) and not w.main_grad.any()


def test_the_optimizer_takes_both(norm):
    """A weight whose gradients are watched ends up where an unwatched one does, but for the rounding of its gradient."""
    from composed_mixture_of_experts_engine_b200.models.moe import RMSNorm
    from composed_mixture_of_experts_engine_b200.ops.optim import build_optimizer

    x, _, _ = norm
    got = []
    for hook in (False, True):
        m = RMSNorm(H, dtype=torch.bfloat16).cuda()
        opt = build_optimizer(m, lr=1e-2)
        if hook:
            m.weight.register_hook(lambda g: None)
        opt.zero_grad()
        m(x).float().pow(2).sum().backward()
        opt.step()
        got.append(opt.state_dict()["groups"]["dense"]["m"].clone())
    assert got[0].any() and torch.allclose(got[0], got[1], rtol=2.0 ** -8, atol=1e-6)
