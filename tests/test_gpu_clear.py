"""The maxima that a launch collects start from zero whatever their memory held, for one run and for many, and for runs without rows."""
import pytest
import torch

from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [1, 3, 64])
def test_maxima_of_runs_start_from_zero(runs):
    from arcquant_b200 import _lib, ops

    k = 256
    counts = [(0, 3, 256, 1)[e % 4] for e in range(runs)]
    first = [256 * e for e in range(runs)]
    x = torch.randn(256 * runs, k, device="cuda").bfloat16()
    groups = torch.tensor(first + counts, dtype=torch.int32, device="cuda")
    out = torch.full((runs,), 1e9, device="cuda")
    rc = _lib.load().arcq_absmax_grouped_bf16(x.data_ptr(), None, groups.data_ptr(), runs, k, out.data_ptr(), ops._stream())
    assert rc == 0
    want = [float(x[f:f + c].abs().max()) if c else 0.0 for f, c in zip(first, counts)]
    assert out.tolist() == want


@pytest.mark.parametrize("rows", [1, 64, 300])      # weight streaming, and CTA pairs
def test_maximum_of_the_swiglu_epilogue_starts_from_zero(rows):
    from arcquant_b200 import _lib, ops

    n, k = 1024 if rows < 128 else 16384, 256
    a = torch.randint(0, 256, (rows, k // 2), dtype=torch.uint8, device="cuda")
    b = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    sfa = torch.full((ops.sf_bytes(rows, k),), 56, dtype=torch.uint8, device="cuda")
    sfb = torch.full((ops.sf_bytes(n, k),), 56, dtype=torch.uint8, device="cuda")
    alpha, c = torch.tensor([1e-3], device="cuda"), torch.empty(rows, n // 2, dtype=torch.bfloat16, device="cuda")
    amax = torch.full((1,), 1e9, device="cuda")
    rc = _lib.load().arcq_matmul_nvfp4_swiglu(a.data_ptr(), b.data_ptr(), sfa.data_ptr(), sfb.data_ptr(), rows, n, k, alpha.data_ptr(),
                                              None, c.data_ptr(), amax.data_ptr(), ops._stream())
    assert rc == 0 and float(amax) == float(c.abs().max()) > 0


def _quantizer(call):
    names = [k[0] for k in launched_kernels(call) if "arcq_quantize_" in k[0]]
    assert len(names) == 1
    return "rows" if "quantize_rows" in names[0] else "ws"


# (which kernel the RMSNorm and the grouped rows take on 148 SMs: the row kernel clears itself, in front of the other a launch does)
@pytest.mark.parametrize("rows, rms, grouped", [(1, "rows", "rows"), (63, "rows", "rows"), (592, "rows", "rows"), (593, "rows", "rows"),
                                                (2000, "rows", "rows"), (3553, "ws", "rows"), (8000, "ws", "ws")])
@pytest.mark.parametrize("clears", [1, 64])
def test_quantizers_clear_for_the_launch_behind_them(rows, rms, grouped, clears):
    from arcquant_b200 import _lib, ops

    k, lib = 1024, _lib.load()
    x, gain = torch.randn(rows, k, device="cuda").bfloat16(), torch.ones(k, device="cuda").bfloat16()
    idx = torch.randperm(k).to(torch.int16).cuda()
    store = torch.full((clears + 2,), 7.0, device="cuda")
    q, sf = ops.rmsnorm_quantize_x(x, gain, 1e-5, idx, 64)
    q2, sf2 = torch.empty_like(q), torch.empty_like(sf)
    assert _quantizer(lambda: ops.rmsnorm_quantize_x(x, gain, 1e-5, idx, 64, clear=store[1:1 + clears])) == rms
    store.fill_(7.0)
    assert lib.arcq_rmsnorm_quantize_x_clear(x.data_ptr(), gain.data_ptr(), 1e-5, idx.data_ptr(), rows, k, 64, q2.data_ptr(), sf2.data_ptr(),
                                             store[1:].data_ptr(), clears, ops._stream()) == 0
    assert torch.equal(q, q2) and store.tolist() == [7.0] + [0.0] * clears + [7.0]
    groups = torch.tensor([0, 256, 0, rows], dtype=torch.int32, device="cuda")          # (the first run is empty)
    src, amax, orders = torch.zeros(256 + (rows + 255) // 256 * 256 + 256, k, device="cuda").bfloat16(), torch.ones(2, device="cuda"), idx.repeat(2, 1)
    src[256:256 + rows] = x
    store.fill_(7.0)
    assert _quantizer(lambda: ops.quantize_grouped_amax(src, None, amax, orders, groups, src.shape[0], 64, clear=store[1:1 + clears])) == grouped
    store.fill_(7.0)
    want = ops.quantize_grouped_amax(src, None, amax, orders, groups, src.shape[0], 64)
    got = ops.quantize_grouped_amax(src, None, amax, orders, groups, src.shape[0], 64, clear=store[1:1 + clears])
    assert torch.equal(want[0][256:256 + rows], got[0][256:256 + rows]) and torch.equal(want[2], got[2])
    assert store.tolist() == [7.0] + [0.0] * clears + [7.0]
