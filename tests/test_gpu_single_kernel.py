"""The single-CTA kernel for 65 rows and more whose 128 x 128 tiles are one wave: both tile widths, their edges in rows and
columns, K of one partial stage up to where a split K takes over; the bias and residual forms have the bits of an addition."""
import ctypes

import pytest
import torch

from tests.helpers import launched_kernels
from tests.test_gpu_skinny import _close, _operands, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,kq,ke,tile", [
    (65, 8, 64, 0, 64), (128, 72, 256, 64, 64), (129, 200, 1984, 64, 64), (256, 4096, 512, 64, 64), (257, 1000, 960, 64, 64),
    (300, 3208, 128, 64, 128), (333, 6144, 1024, 128, 128), (512, 4728, 256, 0, 128), (100, 9472, 192, 64, 64), (100, 9480, 192, 64, 128),
    (128, 4096, 6016, 128, 64), (256, 1024, 10112, 128, 64), (96, 2048, 3008, 64, 64), (97, 136, 3072, 64, 64), (4100, 130 * 4, 192, 0, None), (2000, 1032, 320, 64, 128)])
def test_one_wave_of_single_cta_tiles(m, n, kq, ke, tile):
    from arcquant_b200 import _lib, ops

    a, sfa, sx, b, sfb, sw, _, _, _ = _operands(m, n, kq, ke, m + n)
    kind, bn = ctypes.c_int(-1), ctypes.c_int(-1)
    assert _lib.load().arcq_matmul_plan(m, n, kq + ke, ctypes.byref(kind), ctypes.byref(bn), None) == 0
    name = launched_kernels(lambda: ops.matmul_dev_alpha(a, b, sfa, sfb, sx, sw))[0][0]
    if tile is not None:
        assert kind.value == _lib.GEMM_KIND_SINGLE and bn.value == tile and "arcq_gemm_kernel" in name
    got = ops.matmul_dev_alpha(a, b, sfa, sfb, sx, sw)
    torch.cuda.synchronize()
    assert ops.gemm_poll_error() == 0
    _close(got, _oracle(a, sfa, b, sfb, float(sx * sw)))
    g = torch.Generator().manual_seed(9)
    res = (0.05 * torch.randn((m, n), generator=g)).to(torch.bfloat16).cuda()
    if tile is not None:
        assert torch.equal(ops.matmul_residual(a, b, sfa, sfb, sx, sw, res), res + got)
    bias = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
    assert torch.equal(ops.matmul_dev_alpha(a, b, sfa, sfb, sx, sw, bias), got + bias)
