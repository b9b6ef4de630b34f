"""RMSNorm's backward refills a slot of its shared-memory ring by asynchronous copies once it has read and used the slot's
values: no read of the slot, and no first use of what was read from it, comes after the refill."""

import re

from composed_mixture_of_experts_engine_b200.ops._ext import CSRC_DIR


def test_ring_slots_are_used_before_they_are_refilled():
    text = (CSRC_DIR / "ops.cu").read_text()
    body = text[text.index("rmsnorm_bwd_kernel("):]
    body = body[body.index("cp_async_wait<S - 1>();"):body.index("if (dw_partial)")]
    before, after = body.split("issue(row +", 1)
    assert "*slot(" not in after
    assert sorted(re.findall(r"\*slot\(s, (\d), i\)", before)) == ["0", "1", "2"]
    raw = re.findall(r"(\w+)(?:\[i\])? = \*slot\(", before)  # names that hold a slot's bytes as they were read
    for name in raw:
        assert not re.search(rf"\b{name}\b", after), name
        assert len(re.findall(rf"\b{name}\b", before)) > 1, name
