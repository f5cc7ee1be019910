"""A status of the C side is an ArcqError that carries it, with the extension and without."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extension", [True, False])
def test_the_status_arrives(extension, monkeypatch):
    from arcquant_b200 import _lib, ops

    if not extension:
        monkeypatch.setattr(ops, "_EXT", False)
    assert bool(ops._ext()) == extension
    x, slots = torch.ones(4, 40, device="cuda", dtype=torch.bfloat16), torch.zeros(8, dtype=torch.int64, device="cuda")
    pos, groups = torch.zeros(4, 2, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
    for call in (lambda: ops.route_topk(x, 2),                                   # 40 experts
                 lambda: ops.moe_layout(slots, 65, 256, 65 * 256 + 256),         # 65 runs
                 lambda: ops.absmax_grouped(x[:, :12].contiguous(), None, groups, 1),      # 12 channels
                 lambda: ops.moe_combine(x[:, :12].contiguous(), pos, torch.ones(4, 2, device="cuda", dtype=torch.bfloat16))):
        with pytest.raises(_lib.ArcqError) as e:
            call()
        assert e.value.status == _lib.ERR_BAD_SHAPE and "bad shape" in str(e.value)
    with pytest.raises(_lib.ArcqError) as e:
        ops.rmsnorm_quantize_x(x, x[0].contiguous(), 1e-5, torch.arange(40, dtype=torch.int16, device="cuda"), 0)
    assert e.value.status in (_lib.ERR_BAD_SHAPE, _lib.ERR_UNSUPPORTED_K)
