"""The per-tensor scale of small tensors, whose maximum the quantizer takes itself: around the sizes where a pass of its own takes over,
activations and weights, and values that a maximum has to get right."""
import pytest
import torch

from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu


def _check(x, weight, k):
    from arcquant_b200 import ops

    idx = torch.randperm(k, generator=torch.Generator().manual_seed(k)).to(torch.int16).cuda()
    ke = 64 if k >= 64 else 0
    q, sf, scale = ops.quantize_tensor_scale(x, idx, ke, 16, weight)
    top = (x if weight else x.abs()).float().max()
    assert scale.shape == () and torch.equal(scale.isnan(), top.isnan()) and (bool(top.isnan()) or float(scale) == float(top * (1.0 / 2688.0)))
    if weight:
        want = ops.reorder_quantize_w((x / scale).contiguous(), idx, ke, mode=16)
    else:
        want = ops.reorder_quantize_x(x, idx, ke, mode=16, scale=scale)
    if not bool(top.isnan()):
        assert torch.equal(q, want[0])
        used = ((x.shape[0] + 127) // 128) * (((k + ke) // 16 + 3) // 4) * 512
        rows = torch.arange(x.shape[0], device="cuda")
        c = torch.arange((k + ke) // 16, device="cuda")
        at = ((rows // 128) * (((k + ke) // 16 + 3) // 4))[:, None] * 512 + (c // 4)[None] * 512 + ((rows % 32) * 16 + ((rows // 32) % 4) * 4)[:, None] + (c % 4)[None]
        assert int(at.max()) < used and torch.equal(sf[at], want[1][at])


@pytest.mark.parametrize("weight", [False, True])
@pytest.mark.parametrize("rows, k", [(1, 16), (3, 64), (1, 512), (15, 4096), (64, 1024), (65, 1024), (7, 8208), (1, 14336), (1, 16384), (255, 64), (256, 64),
                                     (257, 64)])
def test_small_tensors(rows, k, weight):
    _around(rows, k, weight)


# (up to 32 loads of eight channels per thread of a CTA)
@pytest.mark.parametrize("weight", [False, True])
@pytest.mark.parametrize("line, k", [(128, 64), (16, 512), (16, 1024), (16, 4096), (16, 5120), (16, 8192), (8, 8208), (8, 14336), (8, 16384)])
def test_around_the_line(line, k, weight):
    from arcquant_b200 import ops

    idx = torch.arange(k, dtype=torch.int16, device="cuda")
    for rows in (line - 1, line, line + 1):
        x = _around(rows, k, weight)
        assert len(launched_kernels(lambda: ops.quantize_tensor_scale(x, idx, 0, 16, weight))) == (1 if rows <= line else 2)


def _around(rows, k, weight):
    x = torch.randn(rows, k, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16).cuda()
    x[rows - 1, k - 1] = -77.0            # the largest magnitude, the smallest value
    x[rows // 2, k // 2] = 33.0
    _check(x, weight, k)
    return x


@pytest.mark.parametrize("weight", [False, True])
@pytest.mark.parametrize("value", [0.0, -0.0, -1.0, -3e-39, float("inf"), float("-inf"), float("nan")])
def test_special_values(value, weight):
    x = torch.full((3, 1024), -2.0 if value != 0.0 else 0.0).to(torch.bfloat16).cuda()
    x[2, 1000] = value
    _check(x, weight, 1024)
