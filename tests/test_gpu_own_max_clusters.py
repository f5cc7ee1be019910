"""A small tensor's maximum by clusters of CTAs in the quantizer's own launch: the bits of the quantizer that is given the maximum, wherever it
lies, in one launch."""
import pytest
import torch

from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu


def _scales(sf, rows, groups):      # those in use of the 512-byte atoms [row % 32][row / 32 % 4][4 groups]
    atoms = (groups + 3) // 4
    return sf.view(-1, atoms, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(-1, 4 * atoms)[:rows, :groups]


# widths of 32 threads, 256, 512 and of two groups a thread; rows at 16 loads a thread and above (clusters), at 40 and below (two
# launches), at 64 and above (two launches); narrow rows (no clusters)
@pytest.mark.parametrize("k, ke, rows", [(16, 16, 511), (16, 0, 513), (512, 16, 8), (512, 0, 9), (512, 48, 32), (528, 16, 11), (528, 48, 32), (4096, 128, 8),
                                         (4096, 64, 9), (4096, 32, 19), (4096, 32, 20), (4096, 0, 32), (4096, 16, 33), (8192, 512, 27), (8208, 16, 5), (14336, 128, 16),
                                         (14336, 256, 17), (16384, 0, 9)])
@pytest.mark.parametrize("is_weight", [False, True])
def test_clusters_find_the_maximum(k, ke, rows, is_weight):
    from arcquant_b200 import ops

    torch.manual_seed(rows)
    x = torch.randn(rows, k, device="cuda").bfloat16()
    idx = torch.randperm(k).to(torch.int16).cuda()
    threads = ((k // 16 if k <= 8192 else (k // 16 + 1) // 2) + 31) // 32 * 32
    call = lambda: ops.quantize_tensor_scale(x, idx, ke, 16, is_weight)
    loads = rows * k / 8 / threads
    assert len(launched_kernels(call)) == (1 if loads <= 32 or (k >= 512 and 40 <= loads <= 64) else 2)
    n = x.numel()
    for at in (None, 0, n // 8 * 5 + 3, n - 1):          # (with the last: the share of the last CTA)
        for v in (77.0, -99.0, float("inf"), float("nan")):
            if at is not None:
                kept = x.view(-1)[at].clone()
                x.view(-1)[at] = v
            q, sf, s = call()
            amax = (x if is_weight else x.abs()).max().float()
            q1, sf1, s1 = ops.quantize_tensor_scale(x, idx, ke, 16, is_weight, amax=amax)
            torch.testing.assert_close(s, s1, rtol=0, atol=0, equal_nan=True)
            if bool(torch.isfinite(s)):
                assert torch.equal(q, q1) and torch.equal(*(_scales(f, rows, (k + ke) // 16) for f in (sf, sf1))), (at, v)
            if at is None:
                break
            x.view(-1)[at] = kept
    assert x.isfinite().all()


def test_under_an_sm_limit():
    """No clusters there: the same bits, with no more CTAs than the limit."""
    from arcquant_b200 import ops

    x, idx = torch.randn(20, 4096, device="cuda").bfloat16(), torch.randperm(4096).to(torch.int16).cuda()
    free = ops.quantize_tensor_scale(x, idx, 128, 16)
    before = ops.set_sm_limit(5)
    try:
        limited = ops.quantize_tensor_scale(x, idx, 128, 16)
        assert all(ctas <= 5 for _, ctas, _ in launched_kernels(lambda: ops.quantize_tensor_scale(x, idx, 128, 16)))
    finally:
        ops.set_sm_limit(before)
    assert torch.equal(free[0], limited[0]) and torch.equal(free[2], limited[2])
    assert torch.equal(_scales(free[1], 20, 264), _scales(limited[1], 20, 264))
