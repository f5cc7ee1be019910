"""The quantizer of many rows at the edges of its warp sets: every width of a set (1 to 8 warps), rows whose last slot and last 32 groups reach back,
critical groups that begin in the middle of 32, no and only critical groups, an odd last row, more pairs than sets, divisors that take the IEEE
division, channel orders off a 16-byte boundary; against the oracle by rows of the first, the middle and the last pairs."""
import numpy as np
import pytest
import torch

from arcquant_b200 import synth
from oracle import oracle as O
from tests.helpers import launched_kernels, sf_take_rows

pytestmark = pytest.mark.gpu


def _sample(rows):
    return sorted({0, 1, 2, 295, 296, 297, 3551, 3552, rows // 2, rows - 2, rows - 1} & set(range(rows)))


@pytest.mark.parametrize("rows, k, ke, mode, form", [
    (9001, 512, 0, 16, "plain"), (9000, 528, 528, 16, "plain"), (9001, 1040, 48, 16, "given"), (8001, 1024, 64, 16, "rms"), (7201, 2048, 256, 16, "rms"),
    (8001, 2048, 128, 32, "own"), (4001, 2064, 16, 16, "plain"), (4003, 4096, 4096, 16, "plain"), (4003, 4096, 1024, 32, "weight"), (3601, 4096, 0, 16, "rms"),
    (4001, 3072, 64, 16, "rms"), (2401, 4112, 80, 16, "given"), (2401, 5120, 128, 16, "rms"), (2401, 6144, 96, 32, "own"), (2001, 6160, 64, 16, "plain"),
    (1801, 7168, 128, 16, "rms"), (2002, 8192, 128, 16, "rms"), (2001, 8192, 8192, 32, "weight"), (1801, 8208, 112, 16, "plain"), (1801, 11008, 64, 16, "own"),
    (1801, 12288, 0, 16, "own"), (1801, 12304, 64, 16, "given"), (1801, 14336, 128, 16, "own"), (1801, 16384, 256, 32, "own")])
def test_against_the_oracle(rows, k, ke, mode, form):
    from arcquant_b200 import ops

    x = synth.activations(rows, k, rows, synth.outlier_channels(k, 20, 1))
    room = torch.zeros(k + 1, dtype=torch.int16, device="cuda")
    order = torch.randperm(k, generator=torch.Generator().manual_seed(k)).to(torch.int16)
    idx = room[rows % 2:rows % 2 + k]             # (odd row counts: two bytes off a 16-byte boundary)
    idx.copy_(order)
    at, xd, gain = _sample(rows), x.cuda(), synth.rms_gain(k, 2, device="cuda")
    call = {"plain": lambda: ops.reorder_quantize_x(xd, idx, ke, mode=mode), "weight": lambda: ops.reorder_quantize_w(xd, idx, ke, mode=mode),
            "rms": lambda: ops.rmsnorm_quantize_x(xd, gain, 1e-5, idx, ke), "own": lambda: ops.quantize_tensor_scale(xd, idx, ke, mode)[:2],
            "given": lambda: ops.reorder_quantize_x(xd, idx, ke, mode=mode, scale=torch.full((), 0.37, device="cuda"))}[form]
    assert "quantize_ws_kernel_sets" in launched_kernels(call)[-1][0]
    q, sf = call()
    scale = {"own": xd.abs().max().float() / 2688.0, "given": torch.full((), 0.37, device="cuda")}.get(form)
    src = x[at] if scale is None else (xd / scale).cpu()[at]
    want, sf_w = O.quantize_w(src, order.numpy(), ke, mode) if form == "weight" else \
        O.quantize_x(src, order.numpy(), ke, mode, gamma=gain.cpu() if form == "rms" else None, eps=1e-5 if form == "rms" else 0.0)
    assert np.array_equal(q.cpu().numpy()[at], want)
    assert np.array_equal(sf_take_rows(sf, at, k + ke), sf_take_rows(sf_w, range(len(at)), k + ke))


@pytest.mark.parametrize("divisor", [0.0, float("inf"), float("nan"), 1e-35, 3e38])
def test_divisors_that_are_no_ordinary_number(divisor):
    from arcquant_b200 import ops

    x = synth.activations(2001, 4096, 5, synth.outlier_channels(4096, 20, 1)).cuda()
    x[7, 11], x[8, 12], x[9, :] = float("inf"), float("nan"), 0.0
    s, idx = torch.tensor(divisor, device="cuda"), torch.randperm(4096).to(torch.int16).cuda()
    many = ops.reorder_quantize_x(x, idx, 64, mode=16, scale=s)
    few = ops.reorder_quantize_x(x[:800], idx, 64, mode=16, scale=s)          # (the row kernel)
    assert torch.equal(many[0][:800], few[0])
    assert np.array_equal(sf_take_rows(many[1], range(800), 4160), sf_take_rows(few[1], range(800), 4160))
