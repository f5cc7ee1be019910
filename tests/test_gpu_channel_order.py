"""The channel order of a statistic against torch's stable sort: it has to place equal values (a statistic is the maximum of
bf16 numbers, so many are equal) in order of their channels, at block and CTA edges too."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 32, 33, 2048, 4095, 4096, 4097, 5120, 8192, 32752])
@pytest.mark.parametrize("values", ["bf16", "constant", "special"])
def test_channel_order_is_a_stable_ascending_sort(k, values):
    from arcquant_b200 import ops

    g = torch.Generator().manual_seed(k)
    if values == "constant":
        v = torch.full((k,), 3.0)
    else:
        v = torch.randn(k, generator=g).abs().to(torch.bfloat16).float()
    if values == "special":
        spots = torch.randint(0, k, (min(k, 40),), generator=g)
        v[spots] = torch.tensor([0.0, -0.0, float("inf"), float("nan"), -1.5, -float("inf"), 1e-40, 448.0]).repeat(5)[: spots.numel()]
    got = ops.channel_order(v.cuda())
    assert got.dtype == torch.int16
    assert torch.equal(got.long().cpu(), torch.sort(v, stable=True).indices)


def test_reorder_index_of_a_calibration():
    from arcquant_b200 import calibrate

    stat = calibrate.ChannelAbsMax()
    for seed in range(3):
        stat.update(torch.randn(200, 4096, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda())
    assert torch.equal(stat.reorder_index().long(), torch.sort(stat.value, stable=True).indices)
