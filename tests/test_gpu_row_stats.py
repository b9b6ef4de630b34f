"""Softmax statistics that the GEMM of the logits leaves, and the cross-entropy that starts from them, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,V,K", [
    (1, 8, 64), (129, 64, 64), (130, 72, 64),   # one piece of columns, one and a bit
    (257, 256, 128), (300, 264, 128),           # one tile, a second one with a single group of eight
    (64, 1000, 64), (700, 8200, 256),
])
def test_stats_and_loss(rows, V, K):
    from composed_mixture_of_experts_engine_b200.ops import _ext, kernels

    g = torch.Generator(device="cuda").manual_seed(rows + V)
    x = torch.randn(rows, K, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(V, K, device="cuda", generator=g).to(torch.bfloat16)
    if V >= 64:  # row 0 holds the columns' numbers as they are: values that the type can just hold, a far maximum, equal ones
        x[0] = 0
        x[0, 0] = 1
        w[:, 0] = torch.linspace(-80, 80, V, device="cuda").to(torch.bfloat16)
        w[8:40, 0] = torch.finfo(torch.bfloat16).min
        w[40:64, 0] = 80
        x[1:, 0] = 0
    ext, status = _ext.ext(), kernels.status_word(x.device)
    y, stats = ext.linear_stats(x, w, status)
    assert torch.equal(y, kernels.linear_nt(x, w)) and stats is not None
    n = (V + 255) // 256
    pad = torch.full((rows, n * 256), float("-inf"), dtype=torch.float64, device="cuda")
    pad[:, :V] = y.double()
    pad = pad.view(rows, n, 256)
    mx = pad.max(2).values
    assert torch.equal(stats[:, :, 0].double(), mx)
    want = (pad - mx[..., None]).exp().sum(2)
    # up to 256 terms of at most 1, each within a few units of fp32 (2^-24) times the exponent's size (160)
    assert float(((stats[:, :, 1].double() - want) / want).abs().max()) <= 160 * 2.0 ** -22
    tgt = torch.randint(0, V, (rows,), device="cuda", generator=g)
    tgt[-1] = -100 if rows > 1 else tgt[-1]
    a, b = y.clone(), y.clone()
    la, lb = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
    ext.cross_entropy(a, tgt, la, 0.5, stats)
    ext.cross_entropy(b, tgt, lb, 0.5)
    live = tgt >= 0
    p = torch.softmax(y.double(), 1)
    p[live.nonzero().flatten(), tgt[live]] -= 1
    p[~live] = 0
    loss = torch.nn.functional.cross_entropy(y.double(), tgt, reduction="sum", ignore_index=-100)
    for grad, l in ((a, la), (b, lb)):
        assert abs(float(l) - float(loss)) <= 1e-5 * max(1.0, abs(float(loss)))
        # one rounding to bf16 (2^-9), and p - 1 where p is near 1 (2^-20 of it left)
        assert float((grad.double() - 0.5 * p).abs().max()) <= 2.0 ** -9 * 0.5 + 1e-6
    kernels.check_status(x.device)


def test_statistics_of_other_logits_are_refused():
    from composed_mixture_of_experts_engine_b200.ops import _ext, kernels

    x = torch.randn(4, 64, device="cuda").to(torch.bfloat16)
    w = torch.randn(16, 64, device="cuda").to(torch.bfloat16)
    y, stats = _ext.ext().linear_stats(x, w, kernels.status_word(x.device))
    bad = stats[:2].contiguous()
    with pytest.raises(RuntimeError, match="statistics"):
        _ext.ext().cross_entropy(y, torch.zeros(4, dtype=torch.int64, device="cuda"), torch.zeros(1, device="cuda"), 1.0, bad)


@pytest.mark.parametrize("n", [8, 2040, 8192, 8200, 1 << 20])
def test_scaled_bf16(n):
    from composed_mixture_of_experts_engine_b200.ops import _ext

    x = torch.randn(n, device="cuda").to(torch.bfloat16)
    s = torch.tensor(0.3719, device="cuda")
    assert torch.equal(_ext.ext().scaled_bf16(x, s), x * s.to(torch.bfloat16))
