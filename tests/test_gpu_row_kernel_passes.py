"""The row kernel where its CTAs take more than one pair of rows: around the line to the kernel of many rows and in between, every
form; rows of the first, a middle and the last passes against the oracle.  (The line is a number of rows per SM: 148 of them here.)"""
import numpy as np
import pytest
import torch

from arcquant_b200 import synth
from oracle import oracle as O
from tests.helpers import launched_kernels, sf_take_rows

pytestmark = pytest.mark.gpu


def _sample(rows):
    return sorted({0, 1, 2, 295, 296, 297, 591, 592, rows // 2, rows - 2, rows - 1} & set(range(rows)))


@pytest.mark.parametrize("rows, k, form", [(888, 4096, "rms"), (889, 4096, "rms"), (1777, 2048, "rms"), (3553, 1024, "rms"), (593, 8192, "rms"),
                                           (591, 5120, "rms"), (1775, 2048, "div"), (1777, 2048, "div"), (592, 7168, "plain"), (594, 5120, "weight"),
                                           (1184, 14336, "plain"), (1185, 14336, "plain"), (592, 14336, "div"), (1185, 14336, "div"),
                                           (700, 16384, "plain"), (333, 11008, "weight"),
                                           # (a few wide rows: their groups shared by up to eight CTAs)
                                           (1, 14336, "div"), (16, 8208, "plain"), (36, 11008, "weight"), (37, 16384, "plain"), (74, 14336, "div"),
                                           (75, 14336, "plain"), (148, 9216, "div"), (149, 14336, "plain")])
def test_passes_of_the_row_kernel(rows, k, form):
    from arcquant_b200 import ops

    ke = 64
    x = synth.activations(rows, k, rows, synth.outlier_channels(k, 20, 1))
    idx = torch.randperm(k, generator=torch.Generator().manual_seed(k)).to(torch.int16)
    at = _sample(rows)
    xd, idd = x.cuda(), idx.cuda()
    if form == "rms":
        gain = synth.rms_gain(k, 2)
        q, sf = ops.rmsnorm_quantize_x(xd, gain.cuda(), 1e-5, idd, ke)
        want, sf_w = O.quantize_x(x[at], idx.numpy(), ke, gamma=gain, eps=1e-5)
    elif form == "div":
        s = (xd.abs().max().float() / 2688.0).reshape(())
        q, sf = ops.reorder_quantize_x(xd, idd, ke, mode=16, scale=s)
        want, sf_w = O.quantize_x((xd / s).cpu()[at], idx.numpy(), ke)
    elif form == "plain":
        q, sf = ops.reorder_quantize_x(xd, idd, ke, mode=16)
        want, sf_w = O.quantize_x(x[at], idx.numpy(), ke)
    else:
        q, sf = ops.reorder_quantize_w(xd, idd, ke, mode=16)
        want, sf_w = O.quantize_w(x[at], idx.numpy(), ke)
    torch.cuda.synchronize()
    assert ops.gemm_poll_error() == 0
    assert np.array_equal(q.cpu().numpy()[at], want)
    assert np.array_equal(sf_take_rows(sf, at, k + ke), sf_take_rows(sf_w, range(len(at)), k + ke))


# (the host knows the rows rounded up to 256: 1776 at 4096 channels and 592 of wider rows are the line)
@pytest.mark.parametrize("counts, k, kernel", [((700, 0, 1075), 4096, "ws"), ((1, 1183, 0, 1), 14336, "ws"), ((257, 2, 300, 33), 8192, "ws"),
                                               ((0, 0, 1776), 4096, "ws"), ((701, 0, 833), 4096, "rows"), ((0, 1535, 0, 1), 4096, "rows"),
                                               ((3,) * 60 + (1001, 0, 0, 353), 4096, "rows"), ((1, 509, 0, 1), 14336, "rows"),
                                               ((255, 0, 257), 14336, "rows"), ((257, 2, 220, 33), 8192, "rows"), ((5, 0, 3323), 2048, "rows")])
def test_passes_over_grouped_rows(counts, k, kernel):
    from arcquant_b200 import ops

    ke, e = 64, len(counts)
    first, at = [], 0
    for c in counts:
        first.append(at)
        at += (c + 255) // 256 * 256
    total, bound = sum(counts), (sum(counts) + 255) // 256 * 256 + 256 * e
    x = synth.activations(total, k, 3, synth.outlier_channels(k, 20, 1), device="cuda")
    row_map = torch.zeros(bound, dtype=torch.int32)
    order = torch.randperm(total, generator=torch.Generator().manual_seed(1)).int()
    n = 0
    for f, c in zip(first, counts):
        row_map[f:f + c] = order[n:n + c]
        n += c
    idx = torch.stack([torch.randperm(k, generator=torch.Generator().manual_seed(i)) for i in range(e)]).to(torch.int16).cuda()
    groups = torch.tensor(first + list(counts), dtype=torch.int32, device="cuda")
    amax = ops.absmax_grouped(x, row_map.cuda(), groups, e)
    rm = row_map.cuda()
    q, sf, scale = ops.quantize_grouped_amax(x, rm, amax, idx, groups, bound, ke)
    torch.cuda.synchronize()
    names = [n[0] for n in launched_kernels(lambda: ops.quantize_grouped_amax(x, rm, amax, idx, groups, bound, ke))]
    assert ["arcq_quantize_rows" in n for n in names] == [kernel == "rows"]
    assert ops.gemm_poll_error() == 0
    for i, (f, c) in enumerate(zip(first, counts)):
        if c == 0:
            continue
        rows = _sample(c)
        src = (x[row_map[f:f + c][rows].long().cuda()] / scale[i]).cpu()
        want, sf_w = O.quantize_x(src, idx[i].cpu().numpy(), ke)
        assert np.array_equal(q.cpu().numpy()[[f + r for r in rows]], want)
        assert np.array_equal(sf_take_rows(sf, [f + r for r in rows], k + ke), sf_take_rows(sf_w, range(len(rows)), k + ke))
