"""SwiGLU of 81 to 128 rows where CTA pairs take over from weight streaming: which kernel, and its result against the separate
SiLU pass, on both sides of the line in rows and in columns."""
import pytest
import torch

from arcquant_b200 import synth
from tests.helpers import launched_kernels
from tests.test_gpu_skinny import _operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,f,kq,pairs", [(80, 3584, 512, False), (81, 3584, 512, True), (128, 9472, 256, True), (128, 9600, 256, False),
                                          (100, 3072, 512, False), (97, 3200, 1024, True)])
def test_swiglu_of_81_to_128_rows(m, f, kq, pairs):
    from arcquant_b200 import ops

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line is a share of the SMs")
    a, sfa, sx, _, _, _, _, _, idx = _operands(m, 16, kq, 64, m)
    wg, wu = synth.weights(f, kq, 5, device="cuda"), synth.weights(f, kq, 6, device="cuda")
    sw = torch.max(torch.cat([wg, wu], 0)).float() / 2688.0
    b1, sfb1 = ops.reorder_quantize_w((torch.cat([wg, wu], 0) / sw).contiguous(), idx, 64)
    b2, sfb2 = ops.reorder_quantize_w((ops.interleave_gate_up(wg, wu) / sw).contiguous(), idx, 64)
    kernels = [name for name, _, _ in launched_kernels(lambda: ops.matmul_swiglu(a, b2, sfa, sfb2, sx, sw))]
    assert any(("arcq_gemm2_kernel" if pairs else "arcq_skinny_kernel") in k for k in kernels)
    want, amax_w = ops.silu_mul(ops.matmul_dev_alpha(a, b1, sfa, sfb1, sx, sw))
    got, amax = ops.matmul_swiglu(a, b2, sfa, sfb2, sx, sw)
    assert ops.gemm_poll_error() == 0
    g, w = got.double(), want.double()
    # fp32 sums of the same products in another order: a bf16 step now and then
    assert float((g - w).norm()) <= 1e-3 * float(w.norm()) and float((got == want).float().mean()) >= 0.99
    assert float(amax) == float(got.abs().max())
