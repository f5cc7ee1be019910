"""The bias in the GEMM's epilogue has the bits of `y + bias` behind it, in every kernel that may serve the shape."""
import pytest
import torch

from arcquant_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,kq", [(1, 8, 64), (16, 4096, 4096), (64, 1000, 1024), (65, 1000, 1024), (333, 4104, 512), (100, 19080, 512),
                                    (1000, 4104, 512), (300, 28672, 512)])
def test_bias_equals_the_addition_behind_the_gemm(m, n, kq):
    from arcquant_b200 import ops

    ke = 64 if kq > 64 else 0
    idx = torch.randperm(kq, generator=torch.Generator().manual_seed(m)).to(torch.int16).cuda()
    a, sfa = ops.reorder_quantize_x(synth.activations(m, kq, 1, synth.outlier_channels(kq, 1, 1), device="cuda"), idx, ke)
    b, sfb = ops.reorder_quantize_w(synth.weights(n, kq, 2, device="cuda"), idx, ke)
    alpha = torch.tensor(0.37, dtype=torch.float32, device="cuda")
    bias = torch.randn(n + 1, generator=torch.Generator().manual_seed(n)).to(torch.bfloat16).cuda()
    y = ops.matmul_dev_alpha(a, b, sfa, sfb, alpha, alpha)
    for v in (bias[:n], bias[1:], bias[:n].float()):               # (off its alignment, fp32: added behind the GEMM)
        got = ops.matmul_dev_alpha(a, b, sfa, sfb, alpha, alpha, v)
        assert got.dtype == (y + v).dtype and torch.equal(got, y + v)
    assert ops.gemm_poll_error() == 0
