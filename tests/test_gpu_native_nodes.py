"""The native autograd nodes against the Python functions of the same operations (which traces and forward-mode calls take):
the same kernels run, so results and gradients have the same bits; also with saved tensors that hooks have moved."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _leaf(g, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16).requires_grad_()


def _linear(g):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    x, w = _leaf(g, 3, 70, 264), _leaf(g, 136, 264)
    return [x, w], lambda: [OF.linear(x, w)]


def _linear_main(g):
    leaves, run = _linear(g)
    leaves[1].main_grad = torch.ones(136, 264, device="cuda")
    return leaves, run


def _linear_frozen(g):
    leaves, run = _linear(g)
    leaves[1].requires_grad_(False)
    return leaves, run


def _norm(g):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    x, w = _leaf(g, 2, 33, 1032), _leaf(g, 1032)
    return [x, w], lambda: list(OF.add_rmsnorm(x, None, w))


def _norm_joined(g):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    x, d, w = _leaf(g, 2, 33, 1032), _leaf(g, 2, 33, 1032), _leaf(g, 1032)
    w.main_grad = torch.ones(1032, device="cuda")
    return [x, d, w], lambda: list(OF.add_rmsnorm(x, d, w))


def _attention(g):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    base = _leaf(g, 2, 100, 12, 64)
    cos, sin = OF.rope_tables(128, 64, 10000.0, torch.device("cuda"))
    return [base], lambda: [OF.rope_causal_attention(base * 1, cos, sin, 4, 4)]


def _router(g):
    from composed_mixture_of_experts_engine_b200.ops.moe_router import MoERouter

    with torch.device("cuda"):
        r = MoERouter(128, 16, 2, dtype=torch.bfloat16)
    r.gate_w.data.normal_(generator=g)
    x = _leaf(g, 300, 128)

    def run():
        idx, w, counts = r(x)
        assert idx.dtype == torch.int64 and int(counts.sum()) == 600 and not idx.requires_grad
        assert r.last_profile.dispatch_counts == counts.tolist()
        return [w, r.last_w32, r.last_aux_loss, r.last_z_loss]

    return [x, r.gate_w], run


def _moe(K, capacity=0):
    def make(g):
        from composed_mixture_of_experts_engine_b200.ops import functional as OF

        x, w13, w2 = _leaf(g, 300, 128), _leaf(g, 8, 144, 128, scale=0.1), _leaf(g, 8, 128, 72, scale=0.1)
        gate = torch.rand(300, K, device="cuda", generator=g).requires_grad_()
        idx = torch.rand(300, 8, device="cuda", generator=g).topk(K, 1).indices
        if capacity:
            w13.main_grad = torch.zeros(8, 144, 128, device="cuda")
        return [x, gate, w13, w2], lambda: [OF.local_moe(x, gate, idx, w13, w2, capacity)]

    return make


CASES = dict(linear=_linear, linear_main=_linear_main, linear_frozen=_linear_frozen, norm=_norm, norm_joined=_norm_joined,
             attention=_attention, router=_router, moe=_moe(2), moe_one_pick=_moe(1), moe_dropping=_moe(2, 40))


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("hooks", [False, True])
def test_nodes_match_the_python_functions(name, hooks, monkeypatch):
    from composed_mixture_of_experts_engine_b200.ops import kernels

    results = []
    for python in (False, True):
        with monkeypatch.context() as m:
            if python:
                m.setattr(kernels, "traced_or_dual", lambda *t: True)
            leaves, run = CASES[name](torch.Generator(device="cuda").manual_seed(3))
            if hooks:
                with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t):
                    outs = run()
            else:
                outs = run()
            assert python == any(type(o.grad_fn).__module__ != "builtins" and "Fn" in type(o.grad_fn).__name__
                                 or "FusedRouter" in type(o.grad_fn).__name__ for o in outs)
            g = torch.Generator(device="cuda").manual_seed(4)
            diff = [o for o in outs if o.requires_grad]
            torch.autograd.backward(diff, [torch.randn(o.shape, device="cuda", generator=g).to(o.dtype) for o in diff])
            results.append([o.detach() for o in outs] + [t.grad for t in leaves] + [getattr(t, "main_grad", None) for t in leaves])
    for a, b in zip(*results):
        assert (a is None) == (b is None) and (a is None or torch.equal(a, b))
    kernels.check_status(torch.device("cuda", 0))


def test_nodes_without_a_gradient():
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    x, w = torch.randn(5, 64, device="cuda").to(torch.bfloat16), torch.randn(8, 64, device="cuda").to(torch.bfloat16)
    assert OF.linear(x, w).grad_fn is None
    with torch.no_grad():
        assert not OF.linear(x.clone().requires_grad_(), w).requires_grad
    y = OF.linear(x.clone().requires_grad_(), w)
    y.sum().backward(retain_graph=True)
    y.sum().backward()  # nothing of the node is used up
