"""Outputs of the extension's calls are allocations that torch can see, trace and fill."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


def _call(rows=3, k=1024):
    from arcquant_b200 import ops

    x, gain = torch.ones(rows, k, device="cuda", dtype=torch.bfloat16), torch.ones(k, device="cuda", dtype=torch.bfloat16)
    idx = torch.arange(k, dtype=torch.int16, device="cuda")
    return lambda: ops.rmsnorm_quantize_x(x, gain, 1e-5, idx, 64)


def test_a_dispatch_mode_sees_them():
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    call = _call()
    want = call()
    with Mode():
        got = call()
    assert seen.count("aten.empty.memory_format") == 2
    assert torch.equal(got[0], want[0])
    seen.clear()
    call()
    assert not seen


def test_deterministic_mode_fills_them():
    call, before, fill = _call(), torch.are_deterministic_algorithms_enabled(), torch.utils.deterministic.fill_uninitialized_memory
    torch.use_deterministic_algorithms(True)
    try:
        torch.utils.deterministic.fill_uninitialized_memory = True
        sf = call()[1]
    finally:
        torch.use_deterministic_algorithms(before)
        torch.utils.deterministic.fill_uninitialized_memory = fill
    # three rows of 68 scales are written; the padding of the tile and the spare one keep torch's fill, the largest byte
    assert int((sf == 255).sum()) == sf.numel() - 3 * 68


@pytest.mark.parametrize("context", [torch.no_grad, torch.inference_mode, lambda: torch.autocast("cuda", torch.bfloat16), torch.enable_grad])
def test_other_contexts_change_nothing(context):
    call = _call()
    want = call()
    with context():
        got = call()
    assert torch.equal(got[0], want[0]) and got[0].is_inference() == (context is torch.inference_mode)
    assert not got[0].requires_grad
