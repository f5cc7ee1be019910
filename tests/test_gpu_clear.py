"""The maxima that a launch collects start from zero whatever their memory held, for one run and for many, and for runs without rows."""
import pytest
import torch

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
