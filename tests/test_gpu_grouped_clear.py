"""`clear` of the grouped quantizer: the same values accepted, refused and set, with the extension, without it, and where torch takes the
scales."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extension", [True, False])
@pytest.mark.parametrize("runs, rows", [(2, 512), (2, 0), (65, 65 * 256)])      # by its maxima; no rows, and more than 64 runs: in torch
def test_clear(runs, rows, extension, monkeypatch):
    from arcquant_b200 import ops

    if not extension:
        monkeypatch.setattr(ops, "_EXT", False)
    k = 512
    x = torch.randn(rows, k, device="cuda").bfloat16()
    groups = torch.tensor([256 * e for e in range(runs)] + [min(rows, 5)] * runs, dtype=torch.int32, device="cuda")
    orders, amax = torch.stack([torch.randperm(k)] * runs).to(torch.int16).cuda(), torch.full((runs,), 4.0, device="cuda")

    def call(clear=None):
        return ops.quantize_grouped_amax(x, None, amax, orders, groups, rows, 64, clear=clear)

    if runs > 64:
        with pytest.raises(RuntimeError):      # (more runs than a launch takes: nothing is set)
            call(torch.ones(2, device="cuda"))
    else:
        store = torch.full((66,), 7.0, device="cuda")
        want, got = call(), call(store[1:65])
        assert torch.equal(want[2], got[2]) and store.tolist() == [7.0] + [0.0] * 64 + [7.0]
        for e in range(runs if rows else 0):
            assert torch.equal(want[0][256 * e:256 * e + 5], got[0][256 * e:256 * e + 5])
    for bad in (torch.ones(65, device="cuda"), torch.ones(2, device="cuda").half(), torch.ones(2), torch.ones(4, device="cuda")[::2]):
        with pytest.raises(RuntimeError):
            call(bad)
        assert bool((bad == 1).all())
    if rows and runs <= 64:
        with pytest.raises(RuntimeError):
            call(amax)
        assert bool((amax == 4).all())
