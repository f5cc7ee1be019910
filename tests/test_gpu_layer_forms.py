"""A half of the decoder layer as one native call and as the operations one by one: the same launches, the same bits."""
import pytest
import torch

from tests.helpers import launched_kernels

pytestmark = pytest.mark.gpu


def _layer(heads, kv_heads, tp=1, rank=0):
    from arcquant_b200.llama_layer import LlamaLayerConfig, QLlamaDecoderLayerTP, random_layer_weights, random_reorder_indices

    cfg = LlamaLayerConfig(hidden=1024, n_heads=heads, n_kv_heads=kv_heads, head_dim=128, ffn=2048, select_num=64)
    return QLlamaDecoderLayerTP(cfg, random_layer_weights(cfg), random_reorder_indices(cfg), rank, tp)


def _halves(layer, x, bsz, pos, residual):
    seq = pos.numel()
    y = layer.attn_partial(x, bsz, seq, pos, residual=x if residual else None)
    return y, layer.mlp_partial(x, residual=x if residual else None)


@pytest.mark.parametrize("heads, kv_heads, tp, rank", [(8, 4, 1, 0), (8, 8, 1, 0), (8, 4, 2, 1)])
@pytest.mark.parametrize("bsz, seq, residual", [(1, 1, True), (3, 1, False), (2, 65, True), (1, 300, False), (1, 4000, True)])
def test_same_bits_and_launches(heads, kv_heads, tp, rank, bsz, seq, residual, monkeypatch):
    from arcquant_b200 import ops

    if residual and tp > 1:
        pytest.skip("the residual is added behind the all-reduce")
    layer = _layer(heads, kv_heads, tp, rank)
    x = torch.randn(bsz * seq, 1024, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seq)).bfloat16()
    pos = torch.arange(seq, device="cuda")
    native = _halves(layer, x, bsz, pos, residual)
    native_names = [k[0] for k in launched_kernels(lambda: _halves(layer, x, bsz, pos, residual), every=True)]
    calls = []
    with monkeypatch.context() as m:
        m.setattr(ops, "attention_half", lambda *a: calls.append(a))
        m.setattr(ops, "mlp_half", lambda *a: calls.append(a))
        m.setattr(ops, "native", lambda: False)
        single = _halves(layer, x, bsz, pos, residual)
        names = [k[0] for k in launched_kernels(lambda: _halves(layer, x, bsz, pos, residual), every=True)]
    assert not calls and names == native_names and len(names) >= 8
    assert all(torch.equal(a, b) for a, b in zip(native, single))


def test_a_timed_step_is_the_untimed_one():
    from arcquant_b200.llama_layer import PhaseTimer

    layer = _layer(8, 4)
    x = torch.randn(2, 65, 1024, device="cuda").bfloat16()
    want = layer(x)
    layer.timer = PhaseTimer()
    got = layer(x)
    times = layer.timer.totals()
    assert torch.equal(got, want) and set(times) == {"quantize", "gemm", "glue", "attention"}


def test_no_rows():
    layer = _layer(8, 4)
    x = torch.empty(0, 1024, device="cuda", dtype=torch.bfloat16)
    assert layer.mlp_partial(x).shape == (0, 1024)


@pytest.mark.parametrize("rows", [1, 64, 300, 4000])
def test_the_cleared_maximum_of_the_public_operators(rows, monkeypatch):
    """rmsnorm_quantize_x(clear) then matmul_swiglu(onto), with the extension and without."""
    from arcquant_b200 import ops

    layer = _layer(8, 4)
    gu, x = layer.gate_up, torch.randn(rows, 1024, device="cuda").bfloat16()
    a, sfa = ops.rmsnorm_quantize_x(x, layer.ln2, 1e-5, gu.index, gu.select_num)
    want = ops.matmul_swiglu(a, gu.W, sfa, gu.SFW, gu.scale)
    for ext in (ops._ext(), False):
        monkeypatch.setattr(ops, "_EXT", ext)
        amax = torch.full((), 1e9, device="cuda")
        a2, sfa2 = ops.rmsnorm_quantize_x(x, layer.ln2, 1e-5, gu.index, gu.select_num, clear=amax)
        got = ops.matmul_swiglu(a2, gu.W, sfa2, gu.SFW, gu.scale, None, amax)
        assert got[1] is amax or got[1].data_ptr() == amax.data_ptr()
        assert torch.equal(a, a2) and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        with pytest.raises(RuntimeError):
            ops.rmsnorm_quantize_x(x, layer.ln2, 1e-5, gu.index, gu.select_num, clear=torch.zeros(65, device="cuda"))
