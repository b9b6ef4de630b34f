"""Embedding gradient where ids repeat: runs that cross the pieces they are cut into, against float64, the same bits on every
run, and no slower than a batch of distinct ids by the length of the run."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def grad(ids, dy, V):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    w = torch.zeros(V, dy.shape[1], device="cuda", dtype=torch.bfloat16).requires_grad_()
    w.main_grad = torch.full((V, dy.shape[1]), 0.25, device="cuda")
    OF.embedding(ids, w).backward(dy)
    return w.main_grad


@pytest.mark.parametrize("runs,H", [
    ([32, 32, 1], 8),              # runs that end with a piece
    ([31, 2, 64, 33], 264),        # across one and two ends of pieces; ragged columns
    ([1, 1000, 1], 136),           # across many pieces, starting and ending inside one
    ([4096], 2048),                # one id fills the batch
    ([5] * 13 + [300] + [1] * 40 + [97], 4104),
])
def test_long_runs(runs, H):
    torch.manual_seed(len(runs))
    V, n = 2 * len(runs) + 1, sum(runs)
    ids = torch.repeat_interleave(torch.arange(len(runs)) * 2 + 1, torch.tensor(runs))[torch.randperm(n)].cuda()
    dy = torch.randn(n, H, device="cuda").to(torch.bfloat16)
    got = grad(ids, dy, V)
    want = torch.full((V, H), 0.25, device="cuda", dtype=torch.float64).index_add(0, ids, dy.double())
    # fp32 sums: each addition rounds by 2^-24 of a partial sum, which stays below 8 sqrt(run) for terms of unit variance;
    # 32 + 8 + pieces / 8 additions deep
    longest = max(runs)
    depth = min(longest, 32) + 8 + longest / 256
    assert float((got.double() - want).abs().max()) <= 2.0 ** -24 * depth * 8 * longest ** 0.5
    assert torch.equal(got, grad(ids, dy, V))
    assert torch.equal(got[0::2], torch.full_like(got[0::2], 0.25))  # rows without a token


def test_one_repeated_id_costs_no_more_than_distinct_ones():
    from composed_mixture_of_experts_engine_b200.ops import _ext

    n, H = 16384, 2048
    dy = torch.randn(n, H, device="cuda").to(torch.bfloat16)
    main = torch.zeros(n, H, device="cuda")
    order = torch.arange(n, device="cuda")

    def us(keys):
        for _ in range(3):
            _ext.ext().embedding_grad(dy, keys, order, main)
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        for _ in range(5):
            _ext.ext().embedding_grad(dy, keys, order, main)
        e[1].record()
        e[1].synchronize()
        return e[0].elapsed_time(e[1]) * 200

    distinct, repeated = us(order), us(torch.full_like(order, 7))
    assert repeated < 3 * distinct, (repeated, distinct)  # reads a fifth of the bytes; in one CTA it took milliseconds
