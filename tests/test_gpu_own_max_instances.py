"""A small tensor's own maximum: which instance of the row kernel takes it - clusters or every CTA, one group a thread or two - and that each gives the
bits of the quantizer that is given the maximum."""
import re

import pytest
import torch

from tests.helpers import launched_kernels
from tests.test_gpu_own_max_clusters import _scales

pytestmark = pytest.mark.gpu


# up to 16 loads a thread every CTA for itself, above that clusters; more than 8192 channels: CTAs that share a pair of rows have one group a thread and
# four chunks, a CTA alone (few SMs) two groups
@pytest.mark.parametrize("rows, k, limit, groups, chunks, clusters", [
    (9, 16, 0, 1, 2, 0), (1, 4096, 0, 1, 2, 0), (8, 4096, 0, 1, 2, 0), (9, 4096, 0, 1, 2, 1), (5, 8192, 0, 1, 2, 0), (11, 8192, 0, 1, 2, 1), (1, 8208, 0, 1, 4, 0),
    (3, 9216, 0, 1, 4, 0), (4, 14336, 0, 1, 4, 0), (5, 14336, 0, 1, 4, 1), (16, 16384, 0, 1, 4, 1), (7, 16384, 8, 1, 4, 0), (7, 16384, 7, 2, 4, 0),
    (8, 9232, 1, 2, 4, 0), (16, 4096, 3, 1, 2, 0)])
def test_each_instance(rows, k, limit, groups, chunks, clusters):
    from arcquant_b200 import ops

    torch.manual_seed(rows + k)
    x, idx, ke = torch.randn(rows, k, device="cuda").bfloat16(), torch.randperm(k).to(torch.int16).cuda(), 16
    want = ops.quantize_tensor_scale(x, idx, ke, 16, amax=x.abs().max().float())
    before = ops.set_sm_limit(limit)
    try:
        kernels = launched_kernels(lambda: ops.quantize_tensor_scale(x, idx, ke, 16))
        got = ops.quantize_tensor_scale(x, idx, ke, 16)
    finally:
        ops.set_sm_limit(before)
    assert len(kernels) == 1 and (limit == 0 or kernels[0][1] <= limit)
    at = [int(v) for v in re.findall(r"L[ib](\d+)E", re.search(r"arcq_quantize_rows_kernelI((?:L[ib]\d+E)+)", kernels[0][0]).group(1))]
    assert (at[0], at[1], at[-2]) == (groups, chunks, clusters), at
    assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
    assert torch.equal(*(_scales(f, rows, (k + ke) // 16) for f in (got[1], want[1])))
