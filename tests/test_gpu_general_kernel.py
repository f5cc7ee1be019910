"""What the general kernel of the quantizer serves: RMSNorm gains off a 16-byte boundary (the bits of aligned ones), rows of more than 16384 channels."""
import numpy as np
import pytest
import torch

from arcquant_b200 import synth
from oracle import oracle as O
from tests.helpers import launched_kernels, sf_take_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, k", [(1, 1024), (37, 4096), (2001, 4096), (5, 4608), (701, 8192)])
def test_gains_off_a_boundary(rows, k):
    from arcquant_b200 import ops

    x, idx, gain = torch.randn(rows, k, device="cuda").bfloat16(), torch.randperm(k).to(torch.int16).cuda(), synth.rms_gain(k, 1, device="cuda")
    off = torch.zeros(k + 8, dtype=torch.bfloat16, device="cuda")[3:3 + k]
    off.copy_(gain)
    call = lambda g: ops.rmsnorm_quantize_x(x, g, 1e-5, idx, 64)
    assert "arcq_quantize_kernel" in launched_kernels(lambda: call(off))[0][0]
    got, want = call(off), call(gain)
    assert torch.equal(got[0], want[0])
    assert np.array_equal(sf_take_rows(got[1], range(rows), k + 64), sf_take_rows(want[1], range(rows), k + 64))


@pytest.mark.parametrize("rows, k, ke, mode", [(3, 16400, 16, 16), (301, 18944, 64, 32), (2, 32752, 0, 16)])
def test_widest_rows(rows, k, ke, mode):
    from arcquant_b200 import ops

    x = synth.activations(rows, k, 1, synth.outlier_channels(k, 20, 1))
    idx = torch.randperm(k, generator=torch.Generator().manual_seed(k)).to(torch.int16)
    q, sf = ops.reorder_quantize_x(x.cuda(), idx.cuda(), ke, mode=mode)
    want, sf_w = O.quantize_x(x, idx.numpy(), ke, mode)
    assert np.array_equal(q.cpu().numpy(), want)
    assert np.array_equal(sf_take_rows(sf, range(rows), k + ke), sf_take_rows(sf_w, range(rows), k + ke))
