"""Scaled weight-gradient output and embedding gradient at the edges of their launch shapes, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 1020, 1024, 4100, 1 << 20])
def test_scaled_out(n):
    from composed_mixture_of_experts_engine_b200.ops import _ext

    torch.manual_seed(n)
    x, s = torch.randn(n, device="cuda"), torch.tensor([0.37], device="cuda")
    acc = torch.randn(n, device="cuda")
    want = acc.double() + float(s) * x.double()
    out = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    _ext.ext().scaled_out(x, s, acc)
    _ext.ext().scaled_out(x, s, out)
    assert torch.allclose(acc.double(), want, rtol=2.0 ** -22, atol=1e-6)
    assert torch.equal(out, (x * s).to(torch.bfloat16))


@pytest.mark.parametrize("B,S,V,H", [(1, 1, 5, 8), (2, 33, 7, 264), (3, 100, 1000, 2048), (1, 50, 9, 4104)])
def test_embedding_gradient_goes_to_main_grad(B, S, V, H):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    torch.manual_seed(H)
    w = torch.randn(V, H, device="cuda").to(torch.bfloat16).requires_grad_()
    w.main_grad = torch.randn(V, H, device="cuda")
    ids = torch.randint(0, V, (B, S), device="cuda")
    ids[0, 0] = V - 1
    dy = torch.randn(B, S, H, device="cuda").to(torch.bfloat16)
    want = w.main_grad.double().index_add(0, ids.flatten(), dy.double().view(-1, H))
    runs = []
    for _ in range(2):
        main = w.main_grad.clone()
        y = OF.embedding(ids, w)
        assert torch.equal(y, torch.nn.functional.embedding(ids, w))
        y.backward(dy)
        assert w.grad is None
        runs.append(w.main_grad.clone())
        w.main_grad.copy_(main)
    assert torch.equal(*runs)
    # fp32 sums of up to S * B terms of size one
    assert float((runs[0].double() - want).abs().max()) <= 2.0 ** -23 * 8 * (1 + B * S / V) * 4
