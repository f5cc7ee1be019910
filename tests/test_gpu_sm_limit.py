"""Under `set_sm_limit(n)` the quantizer and GEMM launches have at most n CTAs - so they occupy at most n SMs, wherever the
scheduler puts them - and give the same results.  Nor do two of them overlap on one stream."""
import ctypes as C

import pytest
import torch

from arcquant_b200 import synth
from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu


def _x(rows, k):
    return synth.activations(rows, k, rows + k, synth.outlier_channels(k, max(1, k // 100), 1), device="cuda")


def _order(k):
    return torch.randperm(k, generator=torch.Generator().manual_seed(k)).to(torch.int16).cuda()


def _quantizers():
    from arcquant_b200 import ops
    from arcquant_b200.qlinear import NVFP4_reorder_quantize_w, NVFP4_reorder_quantize_x

    def rms(rows, k):
        x, idx, gain = _x(rows, k), _order(k), synth.rms_gain(k, 3).cuda()
        return lambda: ops.rmsnorm_quantize_x(x, gain, 1e-5, idx, 64)

    def plain(rows, k):
        x, idx = _x(rows, k), _order(k)
        return lambda: ops.reorder_quantize_x(x, idx, 32)

    def scaled(rows, k, weight=False):
        x, idx = _x(rows, k), _order(k)
        return lambda: (NVFP4_reorder_quantize_w if weight else NVFP4_reorder_quantize_x)(x, idx, 64)

    # the row kernel, the kernel of many rows, narrow rows (the row kernel again), and the kernel of the widest
    return [rms(16, 4096), rms(500, 4096), rms(5000, 4096), rms(3000, 1024), plain(3000, 256), plain(5000, 512), plain(600, 1024),
            plain(5000, 1024), plain(16, 14336), plain(300, 18944), scaled(777, 4096), scaled(16, 14336), scaled(400, 4096, True)]


@pytest.mark.parametrize("limit", [20, 100])
@pytest.mark.parametrize("case", range(13))
def test_quantizers(case, limit):
    from arcquant_b200 import ops

    call = _quantizers()[case]
    want = call()
    before = ops.set_sm_limit(limit)
    try:
        kernels = launched_kernels(call)
        got = call()
    finally:
        ops.set_sm_limit(before)
    torch.cuda.synchronize()
    assert kernels and all("arcq" in name and ctas <= limit for name, ctas, _ in kernels), kernels
    assert torch.equal(got[0], want[0])
    assert all(torch.equal(a, b) for a, b in zip(got[2:], want[2:]))


@pytest.mark.parametrize("k", [1024, 4096])
def test_grouped_quantizer(k):
    """Many rows of runs take a CTA per run at least: a limit below the number of runs is refused.  Few rows go to the row kernel under any limit."""
    from arcquant_b200 import _lib, ops

    runs, ke = 24, 64
    x, orders = _x(runs * 1024, k), torch.stack([torch.randperm(k) for _ in range(runs)]).to(torch.int16).cuda()
    amax = torch.rand(runs, device="cuda") + 3.0

    def call(each):
        groups = torch.tensor([each * i for i in range(runs)] + [each - i for i in range(runs)], dtype=torch.int32, device="cuda")
        return lambda: ops.quantize_grouped_amax(x, None, amax, orders, groups, runs * each, ke)

    few, many = call(256), call(1024)
    want = few()[0], many()[0]
    before = ops.set_sm_limit(runs)
    try:
        kernels, got = launched_kernels(many), many()[0]
        ops.set_sm_limit(runs - 1)
        with pytest.raises(_lib.ArcqError):
            many()
        kernels_few, got_few = launched_kernels(few), few()[0]
    finally:
        ops.set_sm_limit(before)
    assert len(kernels) == 1 and "quantize_ws_kernel_sets" in kernels[0][0] and kernels[0][1] <= runs, kernels
    assert len(kernels_few) == 1 and "quantize_rows_kernel" in kernels_few[0][0] and kernels_few[0][1] < runs, kernels_few
    for each, a, b in ((256, got_few, want[0]), (1024, got, want[1])):
        for i in range(runs):
            assert torch.equal(a[each * i:each * i + each - i], b[each * i:each * i + each - i])


def _packed(rows, k):
    from arcquant_b200 import ops

    return ops.reorder_quantize_x(_x(rows, k), None, 0)


@pytest.mark.parametrize("limit", [20, 100])
@pytest.mark.parametrize("kind,m,n", [("plain", 16, 4096), ("plain", 200, 4096), ("plain", 100, 19200), ("plain", 700, 4096),
                                      ("residual", 333, 1024), ("swiglu", 1, 512), ("swiglu", 16, 28672), ("swiglu", 64, 3584),
                                      ("swiglu", 100, 28672), ("swiglu", 128, 512), ("swiglu", 300, 28672)])
def test_gemms(kind, m, n, limit):
    from arcquant_b200 import ops

    k = 1088
    (a, sfa), (b, sfb) = _packed(m, k), _packed(n, k)
    alpha = torch.tensor(1e-3, device="cuda")
    res = torch.randn((m, n), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    call = {"plain": lambda: ops.matmul_dev_alpha(a, b, sfa, sfb, alpha),
            "residual": lambda: ops.matmul_residual(a, b, sfa, sfb, alpha, None, res),
            "swiglu": lambda: ops.matmul_swiglu(a, b, sfa, sfb, alpha, None)[0]}[kind]
    want = call().double()
    before = ops.set_sm_limit(limit)
    try:
        kernels = launched_kernels(call)
        got = call().double()
    finally:
        ops.set_sm_limit(before)
    assert ops.gemm_poll_error() == 0
    assert kernels and all("arcq" in name and ctas <= limit for name, ctas, _ in kernels), kernels
    # (K may be split differently: an fp32 sum in another order moves an element by one bf16 step now and then)
    assert float((got - want).norm() / want.norm()) <= 1e-3


def _early_starts(fn):
    """Launches that fn() captures as programmatic dependents: edges of the graph of that type."""
    class EdgeData(C.Structure):       # CUgraphEdgeData
        _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]

    cu = C.CDLL("libcuda.so.1")
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    handle, n = C.c_void_p(int(graph.raw_cuda_graph())), C.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(handle, None, None, None, C.byref(n)) == 0
    a, b, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (EdgeData * n.value)()
    assert cu.cuGraphGetEdges_v2(handle, a, b, data, C.byref(n)) == 0
    return sum(d.type == 1 for d in data)      # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC


# of every kernel a launch and, behind it, the ones that could start early: row quantizer and weight streaming; its split form
# behind a maximum; persistent quantizer and CTA pairs, with and without residual; single CTAs; calibration and channel order
@pytest.mark.parametrize("chain", ["decode", "tensor", "prefill", "few", "calibration"])
def test_no_launch_starts_early_under_a_limit(chain):
    from arcquant_b200 import ops

    k, alpha = 1024, torch.tensor(1e-3, device="cuda")
    rows = {"decode": 16, "tensor": 64, "prefill": 4096, "few": 200, "calibration": 300}[chain]
    x, idx, gain = _x(rows, k), _order(k), synth.rms_gain(k, 3).cuda()
    b, sfb = _packed(4096, k)
    res = torch.zeros((rows, 4096), dtype=torch.bfloat16, device="cuda")
    stat, above = torch.zeros(k, device="cuda"), torch.zeros((), dtype=torch.int64, device="cuda")

    def run():
        if chain == "calibration":
            ops.calib_stats(x, stat, above)
            ops.calib_stats(x, stat, above)
            ops.channel_order(stat)
            return
        if chain == "tensor":
            a, sfa, _ = ops.quantize_tensor_scale(x, idx, 0, 16)
        else:
            a, sfa = ops.rmsnorm_quantize_x(x, gain, 1e-5, idx, 0)
        ops.matmul_dev_alpha(a, b, sfa, sfb, alpha)
        ops.matmul_residual(a, b, sfa, sfb, alpha, None, res)

    assert _early_starts(run) >= 2
    before = ops.set_sm_limit(100)
    try:
        limited = _early_starts(run)
    finally:
        ops.set_sm_limit(before)
    assert limited == 0
