"""Calibration that goes on from a caller's own maxima: the count behind the residual width begins with the first batch and goes on whatever the
caller does to `value`."""
import math

import pytest
import torch

from arcquant_b200.calibrate import ChannelAbsMax

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [8, 4096])
@pytest.mark.parametrize("saved", ["before the first batch", "between two batches", "taken away between two batches"])
def test_maxima_of_the_callers(saved, k):
    g = torch.Generator(device="cuda").manual_seed(k)
    batches = [torch.randn(33, k, device="cuda", generator=g).bfloat16() for _ in range(2)]
    own = torch.full((k,), 1.25, device="cuda")
    stat = ChannelAbsMax()
    if saved == "before the first batch":
        stat.value = own.clone()
    stat.update(batches[0])
    if saved == "between two batches":
        stat.value = own.clone()
    if saved == "taken away between two batches":
        stat.value = None
    stat.update(batches[1])
    tops = [b.abs().amax(0).float() for b in batches]
    want = {"before the first batch": torch.maximum(own, torch.maximum(*tops)), "between two batches": torch.maximum(own, tops[1]),
            "taken away between two batches": tops[1]}[saved]
    above = sum(int((b > b.max(dim=-1, keepdim=True)[0] * 0.125).sum()) for b in batches)
    assert torch.equal(stat.value, want)
    assert stat.select_num() == min(math.ceil(k * (above / (66 * k)) / 64) * 64, k)
    assert int(stat._above) == above and stat._seen == 66 * k
