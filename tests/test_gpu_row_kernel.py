"""The row kernel of the quantizer and the per-tensor scale taken inside it: against the oracle, and against the scale
formed in torch followed by the scaled operator.  Codes, scale bytes and the scale itself are exact."""
import numpy as np
import pytest
import torch

from arcquant_b200 import synth
from tests.helpers import launched_kernels, sf_take_rows, valid_sf

pytestmark = pytest.mark.gpu


# narrow rows, one group in the last warp, both sides of 512 groups, odd row counts, and both sides of the row count
# up to which the row kernel runs (444 pairs of rows at 4096 channels, 592 at 14336 on 148 SMs)
@pytest.mark.parametrize("rows,kq,ke", [(1, 16, 16), (3, 64, 0), (5, 528, 16), (33, 1040, 64), (1, 4096, 128), (887, 4096, 128),
                                        (889, 4096, 128), (2, 8192, 256), (3, 8208, 16), (295, 14336, 128), (298, 14336, 64),
                                        (1183, 14336, 128), (1186, 14336, 64),
                                        (7, 16384, 128), (300, 128, 32)])
@pytest.mark.parametrize("weight", [False, True])
def test_tensor_scale_inside_the_quantizer(rows, kq, ke, weight):
    from arcquant_b200 import ops
    from arcquant_b200.qlinear import NVFP4_reorder_quantize_w, NVFP4_reorder_quantize_x
    from oracle import oracle as O

    x = synth.activations(rows, kq, rows + kq, synth.outlier_channels(kq, max(1, kq // 100), 1), device="cuda")
    x[rows // 2, kq // 3] = -x.abs().max() * 3            # the largest magnitude is negative: not a weight's maximum
    idx = torch.randperm(kq, generator=torch.Generator().manual_seed(kq)).to(torch.int16).cuda()
    scale = (x.max() if weight else x.abs().max()).float() / 2688.0
    xs = (x / scale).cpu()
    q, sf, s = (NVFP4_reorder_quantize_w if weight else NVFP4_reorder_quantize_x)(x, idx, ke, mode=16)
    torch.cuda.synchronize()
    assert s.shape == () and torch.equal(s, scale)
    qo, so = (O.quantize_w if weight else O.quantize_x)(xs, idx.cpu().numpy(), ke, mode=16)
    assert np.array_equal(q.cpu().numpy(), qo)
    assert np.array_equal(valid_sf(sf, rows, kq + ke), valid_sf(so, rows, kq + ke))
    if not weight:      # the maximum known beforehand
        q2, sf2, s2 = NVFP4_reorder_quantize_x(x, idx, ke, mode=16, amax=x.abs().max().float())
        assert torch.equal(q2, q) and torch.equal(s2, s)
        assert np.array_equal(valid_sf(sf2, rows, kq + ke), valid_sf(sf, rows, kq + ke))
    assert ops.gemm_poll_error() == 0


@pytest.mark.parametrize("rows,kq", [(1, 1024), (7, 1536), (593, 4096), (590, 4096), (149, 8192), (297, 5120)])
def test_fused_rmsnorm_of_few_rows(rows, kq):
    from arcquant_b200 import ops
    from oracle import oracle as O

    x = synth.activations(rows, kq, rows, synth.outlier_channels(kq, kq // 100, 2), device="cuda")
    gain = synth.rms_gain(kq, 3)
    idx = synth.reorder_index_from_stats(x.abs().amax(0))
    q, sf = ops.rmsnorm_quantize_x(x, gain.cuda(), 1e-5, idx.cuda(), 64)
    qo, so = O.quantize_x(x.cpu(), idx.numpy(), 64, mode=16, gamma=gain, eps=1e-5)
    assert np.array_equal(q.cpu().numpy(), qo)
    assert np.array_equal(valid_sf(sf, rows, kq + 64), valid_sf(so, rows, kq + 64))


@pytest.mark.parametrize("counts,kq", [((1, 0, 5, 2), 4096), ((0, 0, 3, 255), 14336), ((300, 257, 1, 0), 1024), ((3, 0, 0, 2) * 10, 2048)])
def test_grouped_rows_from_the_runs_maxima(counts, kq):
    """Runs with their own maximum, order and divisor equal the per-run calls; an odd run length and an empty run."""
    from arcquant_b200 import _lib, ops
    from arcquant_b200.qlinear import NVFP4_reorder_quantize_x

    e, ke = len(counts), 64
    starts, at = [], 0
    for c in counts:
        starts.append(at)
        at += (c + 255) // 256 * 256
    bound = at + 256
    x = synth.activations(sum(counts), kq, 5, synth.outlier_channels(kq, kq // 100, 2), device="cuda")
    row_map = torch.zeros(bound, dtype=torch.int32)
    src, k = {}, 0
    for i, (s, c) in enumerate(zip(starts, counts)):
        src[i] = torch.arange(k, k + c).flip(0)            # (not the identity)
        row_map[s:s + c] = src[i].int()
        k += c
    groups = torch.tensor(starts + list(counts), dtype=torch.int32, device="cuda")
    idx = torch.stack([torch.randperm(kq, generator=torch.Generator().manual_seed(i)) for i in range(e)]).to(torch.int16).cuda()
    row_map = row_map.cuda()
    amax = ops.absmax_grouped(x, row_map, groups, e)
    q = torch.zeros((bound, (kq + ke) // 2), dtype=torch.uint8, device="cuda")
    sf = torch.zeros((ops.sf_bytes(bound, kq + ke),), dtype=torch.uint8, device="cuda")
    scale = torch.full((e,), -1.0, device="cuda")
    rc = _lib.load().arcq_quantize_x_grouped_amax(x.data_ptr(), row_map.data_ptr(), amax.data_ptr(), idx.data_ptr(), groups.data_ptr(),
                                                  e, bound, kq, ke, 16, q.data_ptr(), sf.data_ptr(), scale.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert torch.equal(scale, amax / 2688.0)
    for i, (s, c) in enumerate(zip(starts, counts)):
        if c == 0:
            continue
        qi, sfi, si = NVFP4_reorder_quantize_x(x[src[i].cuda()].contiguous(), idx[i], ke, mode=16)
        assert torch.equal(si, scale[i])
        assert torch.equal(q[s:s + c], qi)
        run = sf_take_rows(sf, np.arange(s, s + c), kq + ke)
        assert np.array_equal(valid_sf(run, c, kq + ke), valid_sf(sfi, c, kq + ke))


def test_a_weight_off_its_alignment_packs_like_its_copy():
    """A contiguous view at an odd offset of a flat parameter buffer."""
    from arcquant_b200.qlinear import NVFP4_reorder_quantize_w

    n, kq = 130, 1024
    flat = synth.weights(1, n * kq + 8, 3, device="cuda").reshape(-1)
    idx = torch.randperm(kq, generator=torch.Generator().manual_seed(1)).to(torch.int16).cuda()
    for at in (1, 4):
        w = flat[at:at + n * kq].view(n, kq)
        q, sf, s = NVFP4_reorder_quantize_w(w, idx, 64)
        q2, sf2, s2 = NVFP4_reorder_quantize_w(w.clone(), idx, 64)
        assert torch.equal(q, q2) and torch.equal(s, s2)
        assert np.array_equal(valid_sf(sf, n, kq + 64), valid_sf(sf2, n, kq + 64))


@pytest.mark.parametrize("shape", [(), (1,), (1, 1)])
def test_the_scale_has_the_shape_of_the_given_maximum(shape):
    from arcquant_b200.qlinear import NVFP4_reorder_quantize_x

    x = synth.activations(5, 1024, 1, synth.outlier_channels(1024, 10, 1), device="cuda")
    amax = x.abs().max().float().reshape(shape)
    scale = NVFP4_reorder_quantize_x(x, torch.arange(1024, dtype=torch.int16, device="cuda"), 64, amax=amax)[2]
    assert scale.shape == amax.shape and torch.equal(scale, amax / 2688.0)


@pytest.mark.parametrize("rows,widths", [(2, (16384, 14336)), (3000, (2048, 1024)), (3000, (16384, 14336))])
def test_widths_of_one_kernel_from_two_threads(rows, widths):
    """The shared-memory limit belongs to the kernel, not to the thread that raised it: a narrower call of another thread
    must not take it away."""
    from concurrent.futures import ThreadPoolExecutor

    from arcquant_b200 import ops

    def call(kq):
        x = synth.activations(rows, kq, 1, synth.outlier_channels(kq, 10, 1), device="cuda")
        q, _ = ops.reorder_quantize_x(x, torch.arange(kq, dtype=torch.int16, device="cuda"), 64)
        torch.cuda.synchronize()
        return q

    with ThreadPoolExecutor(1) as a, ThreadPoolExecutor(1) as b:
        first = a.submit(call, widths[0]).result()
        b.submit(call, widths[1]).result()
        assert torch.equal(a.submit(call, widths[0]).result(), first)


def test_the_kernel_of_many_rows_keeps_its_values_in_registers():
    """Its 80 registers hold everything, in every instance: shared memory leaves next to no L1, and 100 bytes of spills took plain 16 384 x 4096 from 37 to 45 us."""
    from arcquant_b200 import ops

    met = set()
    for kq in (2048, 4096, 5120, 8192, 11008, 14336):          # rows of up to 128, 256, 320 (384 without RMSNorm), 512, 768 and 1024 groups
        x = synth.activations(3000, kq, 1, synth.outlier_channels(kq, 10, 1), device="cuda")
        idx, one = torch.arange(kq, dtype=torch.int16, device="cuda"), torch.ones((), device="cuda")
        gain = torch.ones(kq, dtype=torch.bfloat16, device="cuda")
        calls = [lambda: ops.reorder_quantize_x(x, idx, 64, scale=one), lambda: ops.quantize_tensor_scale(x, idx, 64), lambda: ops.reorder_quantize_x(x, idx, 64)]
        if kq <= 8192:
            calls += [lambda: ops.rmsnorm_quantize_x(x, gain, 1e-5, idx, 64)]
        for call in calls:
            ws = [k for k in launched_kernels(call) if "quantize_ws_kernel" in k[0]]
            assert len(ws) == 1 and ws[0][2] == 0, ws
            met.add(ws[0][0])
    assert len(met) == 16, sorted(met)                         # (RMSNorm four; six widths, divided and not)
