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


class _Doubled:
    """A linear that is no `PackedLinear`: twice the product of one."""

    def __init__(self, lin):
        self.lin, self.index, self.select_num, self.W, self.SFW, self.scale = lin, lin.index, lin.select_num, lin.W, lin.SFW, lin.scale

    def gemm(self, qx, sfx, scale_x=None, residual=None):
        y = 2 * self.lin.gemm(qx, sfx, scale_x)
        return y if residual is None else residual + y


@pytest.mark.parametrize("name", ["qkv", "o", "down"])
@pytest.mark.parametrize("how", ["instance", "class", "subclass", "module"])
def test_a_linear_of_the_callers_own_is_called(name, how, monkeypatch):
    from arcquant_b200.llama_layer import PackedLinear

    layer = _layer(8, 4)
    x, pos = torch.randn(130, 1024, device="cuda").bfloat16(), torch.arange(65, device="cuda")
    before = _halves(layer, x, 2, pos, False)
    lin, gemm = getattr(layer, name), PackedLinear.gemm
    if how == "instance":
        lin.gemm = lambda *a, **k: 2 * gemm(lin, *a, **k)
    elif how == "class":
        monkeypatch.setattr(PackedLinear, "gemm", lambda self, *a, **k: gemm(self, *a, **k) * (2 if self is lin else 1))
    elif how == "subclass":
        lin.__class__ = type("Own", (PackedLinear,), {"gemm": lambda self, *a, **k: 2 * gemm(self, *a, **k)})
    else:
        delattr(layer, name)
        setattr(layer, name, _Doubled(lin))
    after = _halves(layer, x, 2, pos, False)
    if name == "qkv":       # (twice q, k and v: not twice the output, but another one)
        assert not torch.equal(after[0], before[0]) and torch.equal(after[1], before[1])
    else:
        changed = 0 if name == "o" else 1
        assert torch.equal(after[changed], 2 * before[changed]) and torch.equal(after[1 - changed], before[1 - changed])


def test_parameters_for_buffers():
    layer = _layer(8, 4)
    x, pos = torch.randn(130, 1024, device="cuda").bfloat16(), torch.arange(65, device="cuda")
    before = _halves(layer, x, 2, pos, False)
    for lin in (layer.qkv, layer.o, layer.gate_up, layer.down):
        scale = 2 * lin.scale
        del lin.scale
        lin.scale = torch.nn.Parameter(scale, requires_grad=False)
    after = _halves(layer, x, 2, pos, False)
    assert after[0].shape == before[0].shape and not torch.equal(after[0], before[0]) and not torch.equal(after[1], before[1])


def test_another_attention_is_called(monkeypatch):
    import torch.nn.functional as F
    from torch.overrides import TorchFunctionMode

    layer = _layer(8, 4)
    x, pos = torch.randn(130, 1024, device="cuda").bfloat16(), torch.arange(65, device="cuda")
    want, seen, stock = layer.attn_partial(x, 2, 65, pos), [], F.scaled_dot_product_attention

    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            if func is stock:
                seen.append("mode")
            return func(*args, **(kwargs or {}))

    with Mode():
        assert torch.equal(layer.attn_partial(x, 2, 65, pos), want)
    monkeypatch.setattr(F, "scaled_dot_product_attention", lambda *a, **k: seen.append("replaced") or stock(*a, **k))
    assert torch.equal(layer.attn_partial(x, 2, 65, pos), want)
    assert seen == ["mode", "replaced"]
