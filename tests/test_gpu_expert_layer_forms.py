"""Forms of the expert layer that sizes choose between: rows too wide for the one-pass backward of the combine, and weights
that are read with the hint not to keep them in L2."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K, H, E, F, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(torch.bfloat16)
    x, w13, w2 = mk(N, H), mk(E, 2 * F, H, scale=H ** -0.5), mk(E, H, F, scale=F ** -0.5)
    gate = torch.rand(N, K, device="cuda", generator=g) + 0.5
    idx = torch.rand(N, E, device="cuda", generator=g).topk(K, 1).indices
    return x, gate, idx, w13, w2, mk(N, H)


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("H", [4096, 4104])  # the widest row of the one pass, the first of the two launches
@pytest.mark.parametrize("need_gate", [False, True])
@pytest.mark.parametrize("capacity", [0, 12])
def test_widest_rows(H, need_gate, capacity):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    x, gate, idx, w13, w2, dy = _layer(75, 2, H, 4, 64, H + capacity)
    leaves = [x.requires_grad_(), gate.requires_grad_(need_gate), w13.requires_grad_(), w2.requires_grad_()]
    y = OF.local_moe(x, gate, idx, w13, w2, capacity)
    y.backward(dy)
    exact = [t.detach().double().requires_grad_(t.requires_grad) for t in leaves]
    keep = ~OF.capacity_drop_mask_reference(idx, 4, capacity) if capacity else None
    want = OF.experts_reference(exact[0], idx, exact[1], exact[2], exact[3], 0, keep)
    want.backward(dy.double())
    if capacity:
        assert not keep.all()
        dropped = (~keep).nonzero()
        assert not need_gate or not gate.grad[dropped[:, 0], dropped[:, 1]].any()
    # each value passes up to four roundings to bf16 (rows, gate|up, h, result) of at most 2^-9 each
    assert _rel(y.detach(), want.detach()) <= 2.0 ** -7
    for t, e in zip(leaves, exact):
        assert (t.grad is None) == (e.grad is None) and (t.grad is None or _rel(t.grad, e.grad) <= 2.0 ** -7)
    check_status(x.device)


@pytest.mark.parametrize("N", [40, 1100, 2200])  # narrow tiles of short rows, full tiles, too many rows for the hint
def test_weights_that_are_not_kept(N):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    x, gate, idx, w13, w2, dy = _layer(N, 1, 2048, 16, 704, N)  # 138 MB, more than L2 holds
    with torch.no_grad():
        got = OF.local_moe(x, gate, idx, w13, w2)
        exact = OF.experts_reference(x.double(), idx, gate.double(), w13.double(), w2.double())
    kept = OF.local_moe(x.requires_grad_(), gate, idx, w13, w2).detach()
    assert torch.equal(got, kept) and _rel(got, exact) <= 2.0 ** -7
    check_status(x.device)
