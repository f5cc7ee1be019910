"""A quantized linear finds its weight, scales and bias where they are: registered buffers, replaced ones, or attributes in their place."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [False, True])
def test_where_the_buffers_lie(bias):
    from arcquant_b200.qlinear import NVFP4_reorder_quantize_x, QLinearLayer

    torch.manual_seed(1)
    k, n = 512, 256
    idx = torch.randperm(k).to(torch.int16).cuda()
    make = lambda: QLinearLayer(nn.Linear(k, n, bias=bias, device="cuda", dtype=torch.bfloat16), 64, idx)
    one, other = make(), make()
    x = torch.randn(6, k, device="cuda").bfloat16()
    packed = (*NVFP4_reorder_quantize_x(x, idx, 64), 2, 3)
    want_one, want_other = one(packed), other(packed)
    assert want_one.shape == (2, 3, n) and not torch.equal(want_one, want_other)
    names = ["W", "scale_w", "scale"] + (["bias"] if bias else [])
    for name in names:                                 # assigned: still a buffer
        setattr(one, name, getattr(other, name))
    assert torch.equal(one(packed), want_other)
    for name in names:                                 # a plain attribute, one after the other
        value = getattr(one, name)
        delattr(one, name)
        setattr(one, name, value)
        assert name not in one._buffers and torch.equal(one(packed), want_other)
    state = {name: getattr(make(), name) for name in names}
    third = make()
    want = torch.func.functional_call(third, state, (packed,))
    third.load_state_dict(state)
    assert torch.equal(third(packed), want)
