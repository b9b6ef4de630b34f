"""The decoder joins residual additions with its norms only where calling the modules would do nothing else."""

import pytest
import torch

from composed_mixture_of_experts_engine_b200.models import build_model
from composed_mixture_of_experts_engine_b200.models import decoder as D
from composed_mixture_of_experts_engine_b200.parallel import ParallelTopology
from composed_mixture_of_experts_engine_b200.utils.config import MoEConfig


def _model():
    cfg = MoEConfig.from_dict({
        "model": dict(arch="moe_decoder", hidden_dim=32, num_layers=2, num_heads=2, num_experts=4, top_k=2, ffn_dim=16,
                      vocab_size=64, sequence_length=8, dtype="bfloat16", init_std=0.02),
        "training": dict(micro_batch_size=2), "parallelism": dict(data_parallel=1, expert_parallel=1)})
    return build_model(cfg, ParallelTopology(1, 0, 1, 1, device=torch.device("cpu")))


def _own_forward(m, mp):
    inner = m.forward
    m.forward = lambda x: inner(x) * 2


def _compiled(m, mp):
    m._compiled_call_impl = lambda x: m._call_impl(x) * 2  # what Module.compile() sets


def _patched_class(m, mp):
    inner = type(m).forward
    mp.setattr(type(m), "forward", lambda self, x: inner(self, x) * 2)


def _patched_call(m, mp):
    inner = torch.nn.Module.__call__
    mp.setattr(torch.nn.Module, "__call__", lambda self, *a, **k: inner(self, *a, **k) * (2 if self is m else 1))


def _hook(m, mp):
    m.register_forward_hook(lambda mod, args, out: out * 2)


WATCHERS = [_own_forward, _compiled, _patched_class, _patched_call, _hook]


@pytest.mark.parametrize("watch", WATCHERS)
@pytest.mark.parametrize("where", ["block", "attn_norm", "norm"])
def test_watched_blocks_are_called(watch, where, monkeypatch):
    blk = _model().blocks[0]
    assert blk.joins_residuals()
    watch(blk if where == "block" else getattr(blk, where), monkeypatch)
    assert not blk.joins_residuals()


@pytest.mark.parametrize("watch", WATCHERS)
def test_a_watched_final_norm_is_called(watch, monkeypatch):
    model = _model()
    x, d = torch.randn(2, 8, 32).to(torch.bfloat16), torch.randn(2, 8, 32).to(torch.bfloat16)
    monkeypatch.setattr(model, "_run_blocks", lambda _: (x, d))  # the state in which the last addition would be joined
    monkeypatch.setattr(D.OF, "rmsnorm_supported", lambda *a: False)
    want = model._hidden(x) * 2
    watch(model.norm, monkeypatch)
    assert torch.equal(model._hidden(x), want)


@pytest.mark.parametrize("step", ["run_blocks", "final_hidden"])
@pytest.mark.parametrize("on_class", [False, True])
def test_replaced_steps_are_taken(step, on_class, monkeypatch):
    model = _model()
    seen, inner = [], getattr(D.MoEDecoder, step)
    monkeypatch.setattr(D.MoEDecoder if on_class else model, step,
                        (lambda self, x: (seen.append(1), inner(self, x))[1]) if on_class
                        else lambda x: (seen.append(1), inner(model, x))[1])
    model(torch.randint(0, 64, (1, 8)))
    assert seen == [1]


def test_a_final_norm_in_fp32_is_the_modules_own(monkeypatch):
    """The module rounds its weight to the type of the rows; joined or not, the result has the same bits."""
    model = _model()
    model.norm.weight = torch.nn.Parameter(1 + 0.1 * torch.randn(32))
    x, d = torch.randn(2, 8, 32).to(torch.bfloat16), torch.randn(2, 8, 32).to(torch.bfloat16)
    monkeypatch.setattr(model, "_run_blocks", lambda _: (x, d))
    assert torch.equal(model._hidden(x), model.norm(x + d))
