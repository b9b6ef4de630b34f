"""Calls that bypass an autograd function do so only where nothing asks for it: forward-mode tangents are refused and
traces stay live, as on the path through the function.  The native layer is replaced by stand-ins, so this runs on the
CPU."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD

from composed_mixture_of_experts_engine_b200.ops import functional as OF
from composed_mixture_of_experts_engine_b200.ops import kernels, moe_router

N, H, E, K, F = 6, 8, 8, 2, 4


def fake_router_output(tokens, gate_w, k, timed=False):
    logits = tokens.detach().float() @ gate_w.detach().float()
    w32, idx = torch.topk(torch.softmax(logits, -1), k, -1)
    return moe_router.RouterOutput(idx.to(torch.int32), w32, idx, w32.to(torch.bfloat16), logits,
                                   torch.logsumexp(logits, -1), torch.zeros(E, dtype=torch.int32),
                                   torch.zeros(E, dtype=torch.int64), torch.zeros(E), torch.zeros(4))


class FakeExt:
    def router_route(self, tokens, gate_w, k, full, status):
        o = fake_router_output(tokens, gate_w, k)
        return o.idx32, o.w32, o.idx64, o.w16, o.logits, o.lse, o.counts, o.counts64, o.mean_prob, o.stats


@pytest.fixture
def stand_ins(monkeypatch):
    monkeypatch.setattr(moe_router, "_should_use_fused", lambda *a, **k: True)
    monkeypatch.setattr(moe_router._ext, "ext", lambda: FakeExt())
    monkeypatch.setattr(kernels, "status_word", lambda device: None)
    monkeypatch.setattr(OF, "on_device_path", lambda *t: True)
    monkeypatch.setattr(OF, "_native_forward", lambda x, gate, idx, w13, w2, cap, keep, holder: (x.detach() * 2,) + (None,) * 5)


def calls():
    router = moe_router.MoERouter(H, E, K, dtype=torch.bfloat16).requires_grad_(False)
    gate_w = torch.randn(H, E).to(torch.bfloat16)
    w13, w2 = torch.randn(E, 2 * F, H).to(torch.bfloat16), torch.randn(E, H, F).to(torch.bfloat16)
    gate, idx = torch.rand(N, K), torch.zeros(N, K, dtype=torch.int64)
    return {
        "moe_topk_route": lambda x: moe_router.moe_topk_route(x, gate_w, K)[1],
        "MoERouter": lambda x: router(x)[1],
        "local_moe": lambda x: OF.local_moe(x, gate, idx, w13, w2),
    }


@pytest.mark.parametrize("name", ["moe_topk_route", "MoERouter", "local_moe"])
@pytest.mark.parametrize("grad", [True, False])
def test_forward_mode_is_refused(stand_ins, name, grad):
    x = torch.randn(N, H).to(torch.bfloat16)
    fn = calls()[name]
    with torch.set_grad_enabled(grad):
        fn(x)  # without a tangent the same call is served
        with fwAD.dual_level(), pytest.raises(NotImplementedError):
            fn(fwAD.make_dual(x, torch.ones_like(x)))


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("name,op", [("moe_topk_route", "MoERouterFunction"), ("MoERouter", "FusedRouterFunction"),
                                     ("local_moe", "_NativeLocalMoEFn")])
def test_a_trace_keeps_the_call(stand_ins, name, op):
    x = torch.randn(N, H).to(torch.bfloat16)
    with torch.no_grad():
        traced = torch.jit.trace(calls()[name], (x,), check_trace=False)
    assert f"^{op}" in str(traced.graph)


def embedding_weight():
    w = torch.randn(10, H).to(torch.bfloat16).requires_grad_()
    w.main_grad = torch.zeros(10, H)
    return w


def test_embedding_under_forward_mode(stand_ins):
    w, ids = embedding_weight(), torch.tensor([3, 1, 3])
    with fwAD.dual_level():
        t = torch.randn_like(w)
        y = OF.embedding(ids, fwAD.make_dual(w.detach(), t).requires_grad_())
        assert torch.equal(fwAD.unpack_dual(y).tangent, t[ids])
    dual_w = torch.func.jvp(lambda v: OF.embedding(ids, v), (w.detach(),), (t,))[1]
    assert torch.equal(dual_w, t[ids])


def test_embedding_under_vmap(stand_ins):
    w, ids = embedding_weight(), torch.tensor([[3, 1], [3, 9]])
    assert torch.equal(torch.func.vmap(lambda i: OF.embedding(i, w))(ids), w[ids])


@pytest.mark.filterwarnings("ignore")
def test_embedding_in_a_trace(stand_ins):
    from composed_mixture_of_experts_engine_b200.models.decoder import TokenEmbedding

    emb, ids = TokenEmbedding(10, H, dtype=torch.bfloat16), torch.tensor([3, 1, 3])
    emb.weight.main_grad = torch.zeros(10, H)
    traced = torch.jit.trace(emb, (ids,), check_trace=False)
    assert "aten::embedding" in str(traced.inlined_graph) and torch.equal(traced(ids + 1), emb.weight[ids + 1])
