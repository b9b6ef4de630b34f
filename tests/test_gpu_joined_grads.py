"""Gradients of a decoder whose residual additions are part of its norms, against the same decoder called block by block,
with and without recomputation; a backward pass whose first node is a GEMM on a thread that has touched no GPU yet."""

import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

LAYERS = 3


def _grads(main_grad, watch=(), recompute=False, kv_heads=4):
    from composed_mixture_of_experts_engine_b200.models import build_model
    from composed_mixture_of_experts_engine_b200.ops.optim import build_optimizer
    from composed_mixture_of_experts_engine_b200.parallel import ParallelTopology
    from composed_mixture_of_experts_engine_b200.utils.config import MoEConfig

    cfg = MoEConfig.from_dict({
        "model": dict(arch="moe_decoder", hidden_dim=256, num_layers=LAYERS, num_heads=4, num_kv_heads=kv_heads, num_experts=8,
                      top_k=2, ffn_dim=128, vocab_size=512, sequence_length=64, dtype="bfloat16", init_std=0.05),
        "training": dict(micro_batch_size=2, activation_recompute=recompute),
        "parallelism": dict(data_parallel=1, expert_parallel=1)})
    torch.manual_seed(5)
    model = build_model(cfg, ParallelTopology(1, 0, 1, 1, device=torch.device("cuda", 0)))
    g = torch.Generator().manual_seed(6)
    ids, targets = (torch.randint(0, 512, (2, 64), generator=g).cuda() for _ in range(2))
    for p in model.parameters():
        if p.dim() == 1:  # the norms' weights, all ones
            p.data.add_(0.1 * torch.randn(p.shape, generator=g).to(p))
    if main_grad:
        build_optimizer(model, lr=1e-3)
    for name in watch:
        model.get_submodule(name).register_forward_hook(lambda m, a, out: None)
    loss = model.loss(ids, targets)
    aux, z = model.aux_losses()
    (loss + 0.01 * aux + 0.001 * z).backward()
    got = {n: p.grad if p.grad is not None else p.main_grad for n, p in model.named_parameters()}
    # (recomputation hands the nodes detached weights, whose gradients autograd keeps)
    assert not main_grad or recompute or all(p.grad is None for n, p in model.named_parameters() if not n.endswith("gate_w"))
    return float(loss.detach()), {n: t.detach().double().clone() for n, t in got.items()}


BLOCKS = [f"blocks.{i}" for i in range(LAYERS)]


@pytest.mark.parametrize("main_grad", [False, True])
@pytest.mark.parametrize("kv_heads", [4, 2])
def test_joined_gradients_match_blocks_called_one_by_one(main_grad, kv_heads):
    loss, want = _grads(main_grad, BLOCKS + ["norm"], kv_heads=kv_heads)
    for form in (dict(), dict(watch=["blocks.1.norm"]), dict(watch=BLOCKS[:1]), dict(watch=["norm"]), dict(recompute=True)):
        other, got = _grads(main_grad, kv_heads=kv_heads, **form)
        assert other == loss  # the forward has the same bits
        for n in want:
            # a join adds the two gradients of the stream before it rounds them, which else are rounded one by one: 2^-9 of
            # the norm's part at each of the 2 LAYERS + 1 joins.  A residual's gradient that is lost or counted twice in one
            # place changes what is below it by tens of percent.
            err = float((got[n] - want[n]).norm() / want[n].norm())
            assert err <= (2 * LAYERS + 1) * 2.0 ** -9, (form, n, err)


def test_first_node_of_a_fresh_backward_thread_is_a_gemm():
    """The tensor-map encoder needs a current context, which a thread without a runtime call does not have."""
    code = """
import torch
from composed_mixture_of_experts_engine_b200.ops import functional as OF
x, w, dy = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((64, 128), (256, 128), (64, 256)))
x.requires_grad_(), w.requires_grad_()
OF.linear(x, w).backward(dy)
for got, want in ((x.grad, dy.double() @ w.detach().double()), (w.grad, dy.double().T @ x.detach().double())):
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -8
"""
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
