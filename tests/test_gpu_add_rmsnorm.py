"""Residual addition and RMSNorm in one kernel, both directions, against float64; a decoder whose blocks are watched by
hooks (and so called one by one) against one whose additions are joined."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,H", [(1, 8), (3, 1024), (700, 1032), (5000, 2048), (129, 4104), (9, 8192)])
@pytest.mark.parametrize("join", [False, True])
@pytest.mark.parametrize("main_grad", [False, True])
def test_add_rmsnorm(rows, H, join, main_grad):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    g = torch.Generator(device="cuda").manual_seed(rows + H)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    x, d = mk(rows, H).requires_grad_(), mk(rows, H).requires_grad_() if join else None
    w = (1 + 0.1 * mk(H)).requires_grad_()
    if main_grad:
        w.main_grad = torch.full((H,), 0.5, device="cuda")
    ds, dy = mk(rows, H), mk(rows, H)
    s, y = OF.add_rmsnorm(x, d, w, 1e-5)
    assert torch.equal(s, x + d if join else x)
    sd, wd = s.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    want = sd * torch.rsqrt(sd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    torch.autograd.backward([sd, want], [ds.double(), dy.double()])
    torch.autograd.backward([s, y], [ds, dy])
    rel = lambda a, b: float((a.detach().double() - b.detach()).norm() / b.detach().norm())
    assert rel(y, want) <= 2.0 ** -8 and rel(x.grad, sd.grad) <= 2.0 ** -8  # single roundings to bf16
    if join:
        assert torch.equal(d.grad, x.grad)
    if main_grad:
        assert w.grad is None and rel(w.main_grad - 0.5, wd.grad) <= 1e-5  # fp32 sums (one is added to 0.5)
    else:
        assert rel(w.grad, wd.grad) <= 2.0 ** -8
    # one of the two results unused
    for i in range(2):
        x2 = x.detach().clone().requires_grad_()
        OF.add_rmsnorm(x2, d.detach() if join else None, w.detach(), 1e-5)[i].backward((ds, dy)[i])
        if i == 0:
            assert torch.equal(x2.grad, ds)
        else:
            assert rel(x2.grad, sd.grad - ds.double()) <= 2.0 ** -8


def test_joined_blocks_match_blocks_called_one_by_one():
    from composed_mixture_of_experts_engine_b200.models import build_model
    from composed_mixture_of_experts_engine_b200.parallel import ParallelTopology
    from composed_mixture_of_experts_engine_b200.utils.config import MoEConfig

    cfg = MoEConfig.from_dict({
        "model": dict(arch="moe_decoder", hidden_dim=256, num_layers=3, num_heads=4, num_experts=8, top_k=2, ffn_dim=128,
                      vocab_size=512, sequence_length=64, dtype="bfloat16", init_std=0.02),
        "training": dict(micro_batch_size=2), "parallelism": dict(data_parallel=1, expert_parallel=1)})
    torch.manual_seed(5)
    model = build_model(cfg, ParallelTopology(1, 0, 1, 1, device=torch.device("cuda", 0)))
    ids = torch.randint(0, 512, (2, 64), device="cuda")
    with torch.no_grad():
        joined = model(ids)
        seen = []
        handle = model.blocks[1].norm.register_forward_hook(lambda m, a, out: seen.append(out.shape))
        mixed = model(ids)
        handle.remove()
        handles = [b.register_forward_hook(lambda m, a, out: seen.append(out.shape)) for b in model.blocks]
        called = model(ids)
        for h in handles:
            h.remove()
    assert len(seen) == 4  # every hook has run
    # the additions are rounded at the same places, so the forward has the same bits
    assert torch.equal(joined, mixed) and torch.equal(joined, called)
