"""Up to how many rows the row kernel of the quantizer runs, on both sides of its line, and that the two kernels agree there."""
import pytest
import torch

from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu


def _rows_per_sm(n):
    return n * torch.cuda.get_device_properties(0).multi_processor_count


def _kernel(call):
    names = [k[0] for k in launched_kernels(call) if "arcq_quantize_" in k[0]]
    assert len(names) == 1
    return "rows" if "quantize_rows" in names[0] else "ws"


# (pairs of rows per SM up to which the row kernel serves: x 2 rows)
@pytest.mark.parametrize("k, form, pairs", [(4096, "given", 3), (5120, "given", 1), (8192, "given", 1), (9216, "given", 2), (14336, "given", 2),
                                            (5120, "amax", 2), (14336, "amax", 4), (5120, "plain", 2), (14336, "plain", 4), (2048, "plain", 6),
                                            (8192, "rms", 2), (4096, "rms", 3)])
def test_one_run(k, form, pairs):
    from arcquant_b200 import ops

    at, idx = 2 * _rows_per_sm(pairs), torch.randperm(k).to(torch.int16).cuda()
    x = torch.randn(at + 1, k, device="cuda").bfloat16()
    one, gain = torch.full((), 1.5, device="cuda"), torch.ones(k, device="cuda").bfloat16()

    def call(rows):
        if form == "rms":
            return ops.rmsnorm_quantize_x(x[:rows], gain, 1e-5, idx, 64)
        if form == "amax":
            return ops.quantize_tensor_scale(x[:rows], idx, 64, 16, amax=one)
        return ops.reorder_quantize_x(x[:rows], idx, 64, mode=16, scale=one if form == "given" else None)

    assert _kernel(lambda: call(at)) == "rows" and _kernel(lambda: call(at + 1)) == "ws"
    assert torch.equal(call(at)[0], call(at + 1)[0][:at])


@pytest.mark.parametrize("k, pairs", [(4096, 6), (8192, 2), (9216, 2), (14336, 2)])
def test_eight_runs(k, pairs):
    from arcquant_b200 import ops

    e = 8
    at = 2 * _rows_per_sm(pairs) // 256 * 256                  # the host's bound of the rows: whole tiles
    each = at // e - 1
    first = [i * ((each + 255) // 256 * 256) for i in range(e)]
    bound, more = at + 256 * e, at + 256 * e + 512
    src = torch.randn(max(more, first[-1] + each), k, device="cuda").bfloat16()
    groups = torch.tensor(first + [each] * e, dtype=torch.int32, device="cuda")
    amax, orders = torch.full((e,), 5.0, device="cuda"), torch.stack([torch.randperm(k) for _ in range(e)]).to(torch.int16).cuda()
    row_map = torch.arange(more, dtype=torch.int32, device="cuda")

    def call(rows_bound):
        return ops.quantize_grouped_amax(src, row_map, amax, orders, groups, rows_bound, 64)

    assert first[-1] + each <= bound
    assert _kernel(lambda: call(bound)) == "rows" and _kernel(lambda: call(more)) == "ws"
    a, b = call(bound)[0], call(more)[0]
    for f in first:
        assert torch.equal(a[f:f + each], b[f:f + each])
