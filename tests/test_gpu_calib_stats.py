"""Calibration statistics at the edges of the kernel's groups of rows and of its staged running maxima, against torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])                   # running maxima on a 16-byte boundary, and off it
@pytest.mark.parametrize("rows, k", [(1, 8), (64, 4096), (65, 4096), (73, 4096), (2369, 512), (2401, 4096), (67, 4104), (130, 8192),
                                     (5, 16384), (70, 16392), (9, 32768)])
def test_statistics_of_two_batches(rows, k, shift):
    from arcquant_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows + k)
    batches = [torch.randn(rows, k, device="cuda", generator=g).bfloat16() for _ in range(2)]
    batches[1][rows // 2, k - 1] = -90.0                     # a record in the second batch
    store, above = torch.zeros(k + 4, device="cuda"), torch.zeros((), dtype=torch.int64, device="cuda")
    value = store[shift:shift + k]
    for x in batches:
        ops.calib_stats(x, value, above)
    want = torch.stack([x.abs().amax(0) for x in batches]).amax(0).float()
    count = sum(int((x > x.max(dim=-1, keepdim=True)[0] * 0.125).sum()) for x in batches)
    assert torch.equal(value, want) and int(above) == count
    assert float(store[shift + k:].abs().sum()) == 0 and (shift == 0 or float(store[0]) == 0)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("rows, k", [(1190, 8192), (595, 16384), (299, 16392), (301, 32768)])      # some CTAs take a second step
def test_statistics_of_more_steps_than_ctas(rows, k, shift):
    from arcquant_b200 import ops

    x = torch.randn(rows, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(k)).bfloat16()
    x[rows - 1, 0], x[rows - 2, k - 1], x[0, 7] = 77.0, -99.0, float("-inf")
    x[:, 5] = -0.0
    store, above = torch.zeros(k + 4, device="cuda"), torch.zeros((), dtype=torch.int64, device="cuda")
    value = store[shift:shift + k]
    value[3] = 55.0                                          # a record of an earlier batch
    ops.calib_stats(x, value, above)
    want = x.abs().amax(0).float()
    want[3] = 55.0
    assert torch.equal(value, want) and int(above) == int((x > x.max(dim=-1, keepdim=True)[0] * 0.125).sum())
    assert float(store[shift + k:].abs().sum()) == 0 and (shift == 0 or float(store[0]) == 0)
