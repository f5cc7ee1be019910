"""What the row kernel does by the way - clearing maxima, taking the maximum of a small tensor - is compiled into instances of their own:
launches that ask for neither run the code that has neither."""
import re

import pytest
import torch

from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu
NOTHING, CLEAR, OWN_MAX = "0", "1", "2"


def _by_the_way(call):
    names = [k[0] for k in launched_kernels(call) if "arcq_quantize_rows_kernel" in k[0]]
    assert len(names) == 1
    return re.findall(r"L[ib](\d+)E", re.search(r"arcq_quantize_rows_kernelI((?:L[ib]\d+E)+)", names[0]).group(1))[-1]


@pytest.mark.parametrize("rows, k", [(1, 1024), (16, 4096), (40, 5120), (3, 14336)])      # 256 threads, 512, two groups per thread
def test_only_launches_that_ask_for_it(rows, k):
    from arcquant_b200 import ops

    x = torch.randn(rows, k, device="cuda").bfloat16()
    idx, one = torch.randperm(k).to(torch.int16).cuda(), torch.ones((), device="cuda")
    assert _by_the_way(lambda: ops.reorder_quantize_x(x, idx, 64, mode=16)) == NOTHING
    assert _by_the_way(lambda: ops.reorder_quantize_w(x, idx, 64, mode=16)) == NOTHING
    assert _by_the_way(lambda: ops.reorder_quantize_x(x, idx, 64, mode=16, scale=one)) == NOTHING
    assert _by_the_way(lambda: ops.quantize_tensor_scale(x, idx, 64, 16, amax=one)) == NOTHING
    assert _by_the_way(lambda: ops.quantize_tensor_scale(x, idx, 64, 16)) == (OWN_MAX if rows < 40 else NOTHING)
    src = torch.randn(512, k, device="cuda").bfloat16()
    groups, amax, orders = torch.tensor([0, rows], dtype=torch.int32, device="cuda"), torch.ones(1, device="cuda"), idx[None]
    assert _by_the_way(lambda: ops.quantize_grouped_amax(src, None, amax, orders, groups, 512, 64)) == NOTHING
    clear = torch.ones(3, device="cuda")
    assert _by_the_way(lambda: ops.quantize_grouped_amax(src, None, amax, orders, groups, 512, 64, clear=clear)) == CLEAR
    assert not clear.any()
