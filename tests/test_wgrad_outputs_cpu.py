"""Weight-gradient outputs of every layout: what the kernels can write goes to them, everything else takes the fp32 result by
an ordinary copy or addition.  The native call is replaced by a stand-in that insists on its contract."""

import pytest
import torch

from composed_mixture_of_experts_engine_b200.ops import kernels

R, M, N = 96, 24, 16


class Contract:
    def __init__(self):
        self.calls = []

    def wgrad(self, a, b, out, accumulate, status, pieces):
        assert out.stride(1) == 1 and out.data_ptr() % 16 == 0 and out.stride(0) * out.element_size() % 16 == 0
        assert out.dtype == torch.float32 or (out.dtype == torch.bfloat16 and not accumulate)
        self.calls.append((out.data_ptr(), pieces))
        res = a.float().t() @ b.float()
        if accumulate:
            out.add_(res)
        else:
            out.copy_(res)


def outputs():
    buf = torch.zeros(M * N + 8)
    return {
        "contiguous": torch.zeros(M, N),
        "row stride": torch.zeros(M, N + 4)[:, :N],
        "odd row stride": torch.zeros(M, N + 1)[:, :N],
        "misaligned": buf[1:1 + M * N].view(M, N),
        "transposed": torch.zeros(N, M).t(),
        "bf16": torch.zeros(M, N, dtype=torch.bfloat16),
        "fp64": torch.zeros(M, N, dtype=torch.float64),
    }


@pytest.mark.parametrize("name", list(outputs()))
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("entry", ["linear_tn", "linear_tn_acc"])
def test_every_output_layout_is_served(monkeypatch, name, accumulate, entry):
    ext = Contract()
    monkeypatch.setattr(kernels._ext, "ext", lambda: ext)
    monkeypatch.setattr(kernels, "status_word", lambda device: None)
    torch.manual_seed(0)
    a, b = torch.randn(R, M).to(torch.bfloat16), torch.randn(R, N).to(torch.bfloat16)
    out = outputs()[name].fill_(0.5)
    want = (a.float().t() @ b.float()).to(out.dtype)
    want = want + out if accumulate else want
    got = getattr(kernels, entry)(a, b, out, accumulate)
    assert got is out and torch.equal(out, want)
    in_place = name in ("contiguous", "row stride") or (name == "bf16" and not accumulate)
    assert (ext.calls[0][0] == out.data_ptr()) == in_place


def test_explicit_pieces_and_types(monkeypatch):
    ext = Contract()
    monkeypatch.setattr(kernels._ext, "ext", lambda: ext)
    monkeypatch.setattr(kernels, "status_word", lambda device: None)
    a, b = torch.randn(R, M).to(torch.bfloat16), torch.randn(R, N).to(torch.bfloat16)
    assert kernels.linear_tn(a, b, None, False, 3).dtype == torch.float32
    assert kernels.linear_tn(a, b, splits=2, out_dtype=torch.bfloat16).dtype == torch.bfloat16
    assert [p for _, p in ext.calls] == [3, 2]
