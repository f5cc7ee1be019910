"""The work whose time this library is judged by: calls of its public entry points, over the sizes that a
program which serves or prepares a quantized model uses.

Kinds of case, in the order in which such a program meets them:

  calibrate    running channel statistics over a calibration set, then the channel order and residual width
  pack         one bf16 weight matrix into codes, scales and its global scale (once per matrix and model load)
  quantize     RMSNorm + channel order + NVFP4 of a batch of tokens, alone: the input of several projections
  norm_linear  the same followed by the projection it feeds: the first half of an attention or MLP block
  linear       a quantized linear whose input has no norm in front: global scale of the tensor, quantize, GEMM
  layer        a whole decoder layer, prefill or one token per sequence, eager or as a replayed CUDA graph
  moe          a whole sparse-MoE block

Sizes are the projections of the Llama-3-8B layer and of the Mixtral MoE block that the benchmark runs, their
row-parallel shards, and the other row widths of the reference's operators.
"""
import math

import torch

from arcquant_b200 import graphs, ops, synth
from arcquant_b200.calibrate import ChannelAbsMax
from arcquant_b200.llama_layer import LlamaLayerConfig, PackedLinear, QLlamaDecoderLayerTP
from arcquant_b200.moe_block import MoEConfig, QMixtralMoEBlockEP
from arcquant_b200.qlinear import NVFP4_reorder_quantize_w, NVFP4_reorder_quantize_x, QLinearLayer

EPS = 1e-5
HIDDEN, HEADS, KV_HEADS, HEAD_DIM, FFN = 4096, 32, 8, 128, 14336
EXPERTS, TOP_K = 8, 2
# (in, out) of the projections; the row-parallel shards of two and four ranks behind them
NORM_SHAPES = [(4096, 6144), (4096, 28672), (2048, 3072), (3072, 5120), (5120, 5120), (8192, 10240)]
LINEAR_SHAPES = [(4096, 4096), (4096, 6144), (4096, 28672), (14336, 4096), (7168, 4096), (3584, 4096), (2048, 4096),
                 (5120, 5120), (11008, 4096)]
NORM_WIDTHS = [2048, 3072, 3584, 4096, 5120, 8192]
RESIDUALS = [64, 128, 256]


def listed():
    return [
        # one sequence being decoded: a single token into the fused q/k/v projection; latency and launches count
        dict(name="norm_linear_1_qkv", kind="norm_linear", rows=1, k=4096, n=6144, ke=128),
        # sixteen sequences being decoded, the widest input: weight streaming
        dict(name="linear_16_down", kind="linear", rows=16, k=14336, n=4096, ke=128, bias=False),
        # a short prompt of ragged length, a projection with a bias
        dict(name="linear_777_o", kind="linear", rows=777, k=4096, n=4096, ke=128, bias=True),
        # a prefill chunk into the fused q/k/v projection
        dict(name="norm_linear_4096_qkv", kind="norm_linear", rows=4096, k=4096, n=6144, ke=128),
        # the activation operator alone on a large prefill
        dict(name="quantize_32768", kind="quantize", rows=32768, k=4096, ke=128),
        # a calibration set of 16 sequences, ragged
        dict(name="calibrate_16x2000", kind="calibrate", batches=16, rows=2000, k=4096),
        # one gate matrix of a model being loaded
        dict(name="pack_14336x4096", kind="pack", n=14336, k=4096, ke=128),
        # one decoder layer, one token of sixteen sequences, as a serving loop replays it
        dict(name="layer_16x1_graph", kind="layer", batch=16, seq=1, ke=128, graph=True),
        # one decoder layer, a single ragged prompt, eager
        dict(name="layer_1x333", kind="layer", batch=1, seq=333, ke=128, graph=False),
        # one decoder layer, the benchmark's prefill
        dict(name="layer_8x2048", kind="layer", batch=8, seq=2048, ke=128, graph=False),
        # a sparse-MoE block on the tokens of a decode step: every expert has a handful of rows
        dict(name="moe_37", kind="moe", rows=37, ke=128, graph=False),
        # a sparse-MoE block, the benchmark's prefill
        dict(name="moe_4096", kind="moe", rows=4096, ke=128, graph=False),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["norm_linear", "linear", "layer", "moe", "quantize", "pack", "calibrate"],
                       weights=[5, 6, 5, 4, 3, 1, 1])[0]
    ke = rng.choice(RESIDUALS)
    if kind == "norm_linear":
        k, n = rng.choice(NORM_SHAPES)
        return dict(kind=kind, rows=_log_int(rng, 1, 8192), k=k, n=n, ke=ke)
    if kind == "linear":
        k, n = rng.choice(LINEAR_SHAPES)
        return dict(kind=kind, rows=_log_int(rng, 1, 8192), k=k, n=n, ke=ke, bias=rng.random() < 0.3)
    if kind == "layer":
        if rng.random() < 0.4:      # one token of every sequence
            return dict(kind=kind, batch=_log_int(rng, 1, 256), seq=1, ke=ke, graph=rng.random() < 0.6)
        batch = _log_int(rng, 1, 8)
        return dict(kind=kind, batch=batch, seq=_log_int(rng, 16, 14000 // batch if batch > 6 else 2048), ke=ke,
                    graph=False)
    if kind == "moe":
        rows = _log_int(rng, 1, 4096)
        return dict(kind=kind, rows=rows, ke=ke, graph=rows <= 256 and rng.random() < 0.5)
    if kind == "quantize":          # whole scale tiles: every byte of the returned buffers' used part is written
        return dict(kind=kind, rows=128 * _log_int(rng, 1, 200), k=rng.choice(NORM_WIDTHS), ke=ke)
    if kind == "pack":
        k, n = rng.choice([(4096, 4096), (4096, 14336), (14336, 4096), (5120, 5120), (8192, 10240)])
        return dict(kind=kind, n=n, k=k, ke=ke)
    return dict(kind="calibrate", batches=rng.randint(4, 16), rows=rng.randint(200, 2048),
                k=rng.choice([2048, 4096, 5120, 8192]))


# ---------------------------------------------------------------------------------------------- inputs


def _activations(rows, k, seed):
    """bf16 [rows, k] ~ N(0,1), 1 % of the channels scaled by 50, and the channel order of its statistics."""
    x = synth.activations(rows, k, seed, synth.outlier_channels(k, max(1, k // 100), seed), device="cuda")
    return x, synth.reorder_index_from_stats(x.abs().amax(0)).cuda()


def _weight(n, k, seed):
    return synth.weights(n, k, seed, device="cuda")


def _order(k, seed):
    return torch.randperm(k, generator=torch.Generator().manual_seed(seed)).to(torch.int16)


def _graphed(step, x):
    """A step captured over a static input tensor, as a serving loop keeps it."""
    static = x.clone()
    step(static)
    torch.cuda.synchronize()
    return static, graphs.GraphedStep(lambda: step(static))


def prepare(case, seed):
    kind, s = case["kind"], 1000 * (seed % 1000003)
    st = dict(case=case)
    if kind == "calibrate":
        out = synth.outlier_channels(case["k"], case["k"] // 100, s)
        st["x"] = [synth.activations(case["rows"], case["k"], s + 1 + b, out, device="cuda") for b in range(case["batches"])]
    elif kind == "pack":
        st["w"], st["index"] = _weight(case["n"], case["k"], s), _order(case["k"], s).cuda()
    elif kind in ("quantize", "norm_linear"):
        st["x"], st["index"] = _activations(case["rows"], case["k"], s)
        st["gain"] = synth.rms_gain(case["k"], s + 1, device="cuda")
        if kind == "norm_linear":
            st["lin"] = PackedLinear(_weight(case["n"], case["k"], s + 2), st["index"], case["ke"])
    elif kind == "linear":
        st["x"], st["index"] = _activations(case["rows"], case["k"], s)
        lin = torch.nn.Linear(case["k"], case["n"], bias=case["bias"], device="cuda", dtype=torch.bfloat16)
        lin.weight.data.copy_(_weight(case["n"], case["k"], s + 2))
        if case["bias"]:
            lin.bias.data.copy_(_weight(1, case["n"], s + 3)[0])
        st["lin"] = QLinearLayer(lin, case["ke"], st["index"])
    elif kind == "layer":
        cfg = LlamaLayerConfig(hidden=HIDDEN, n_heads=HEADS, n_kv_heads=KV_HEADS, head_dim=HEAD_DIM, ffn=FFN,
                               select_num=case["ke"], eps=EPS)
        tokens = case["batch"] * case["seq"]
        x, index = _activations(tokens, HIDDEN, s)
        kv = KV_HEADS * HEAD_DIM
        weights = {name: _weight(n, k, s + 10 + i) for i, (name, n, k) in enumerate([
            ("wq", HIDDEN, HIDDEN), ("wk", kv, HIDDEN), ("wv", kv, HIDDEN), ("wo", HIDDEN, HIDDEN),
            ("w_gate", FFN, HIDDEN), ("w_up", FFN, HIDDEN), ("w_down", HIDDEN, FFN)])}
        weights["ln1"] = synth.rms_gain(HIDDEN, s + 20, device="cuda")
        weights["ln2"] = synth.rms_gain(HIDDEN, s + 21, device="cuda")
        indices = {"q": index, "up": index, "o": _order(HIDDEN, s + 22), "down": _order(FFN, s + 23)}
        st["layer"] = layer = QLlamaDecoderLayerTP(cfg, weights, indices)
        st["x"] = x.reshape(case["batch"], case["seq"], HIDDEN)
        st["positions"] = torch.arange(case["seq"], device="cuda")
        if case["graph"]:
            st["static"], st["step"] = _graphed(lambda t: layer(t, st["positions"]), st["x"])
    else:
        cfg = MoEConfig(hidden=HIDDEN, ffn=FFN, n_experts=EXPERTS, top_k=TOP_K, select_num=case["ke"])
        st["x"], index = _activations(case["rows"], HIDDEN, s)
        experts = [{"w1": _weight(FFN, HIDDEN, s + 30 + e), "w3": _weight(FFN, HIDDEN, s + 50 + e),
                    "w2": _weight(HIDDEN, FFN, s + 70 + e), "w1_index": index, "w2_index": _order(FFN, s + 90 + e)}
                   for e in range(EXPERTS)]
        router = _weight(EXPERTS, HIDDEN, s + 5)
        st["block"] = block = QMixtralMoEBlockEP(cfg, {"router": router, "experts": experts})
        if case["graph"]:
            st["static"], st["step"] = _graphed(block, st["x"])
    return st


# ---------------------------------------------------------------------------------------------- one pass


def _used(sf, rows, k_eff):
    """The scale tiles of the rows (the buffer ends with a spare tile, as the reference's does)."""
    return sf[:((rows + 127) // 128) * ((k_eff // 16 + 3) // 4) * 512]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "calibrate":
        stats = ChannelAbsMax()
        for x in st["x"]:
            stats.update(x)
        return stats.value, stats.reorder_index(), stats.select_num()
    if kind == "pack":
        w, sf, scale = NVFP4_reorder_quantize_w(st["w"], st["index"], case["ke"])
        return w, _used(sf, case["n"], case["k"] + case["ke"]), scale
    if kind == "quantize":
        q, sf = ops.rmsnorm_quantize_x(st["x"], st["gain"], EPS, st["index"], case["ke"])
        return q, _used(sf, case["rows"], case["k"] + case["ke"])
    if kind == "norm_linear":
        q, sf = ops.rmsnorm_quantize_x(st["x"], st["gain"], EPS, st["index"], case["ke"])
        return st["lin"].gemm(q, sf)
    if kind == "linear":
        q, sf, scale = NVFP4_reorder_quantize_x(st["x"], st["index"], case["ke"])
        return st["lin"]((q, sf, scale, 1, case["rows"]))
    if case["graph"]:
        st["static"].copy_(st["x"])
        return st["step"]()
    if kind == "layer":
        return st["layer"](st["x"], st["positions"])
    return st["block"](st["x"])


# ---------------------------------------------------------------------------------------------- what it needs


def _packed(rows, k_eff):
    return rows * k_eff * 9 // 16        # codes and block scales


def _gemm(rows, n, k_eff):
    return 2.0 * rows * n * k_eff


def work(case):
    """Bytes: inputs and weights read once, results written once.  Flops: the products over the augmented width."""
    kind = case["kind"]
    if kind == "calibrate":
        elems = case["batches"] * case["rows"] * case["k"]
        return {"bytes": 2 * elems + 4 * case["k"], "flops": 0}
    k = case.get("k", HIDDEN)
    ke = case["ke"]
    if kind == "pack":
        return {"bytes": 2 * case["n"] * k + 2 * k + _packed(case["n"], k + ke), "flops": 0}
    rows = case["batch"] * case["seq"] if kind == "layer" else case["rows"]
    if kind == "quantize":
        return {"bytes": 2 * rows * k + 4 * k + _packed(rows, k + ke), "flops": 0}
    if kind in ("norm_linear", "linear"):
        n = case["n"]
        return {"bytes": 2 * rows * k + 4 * k + _packed(n, k + ke) + 2 * rows * n, "flops": _gemm(rows, n, k + ke)}
    if kind == "layer":
        kv = KV_HEADS * HEAD_DIM
        shapes = [(HIDDEN + 2 * kv, HIDDEN + ke), (HIDDEN, HIDDEN + ke), (2 * FFN, HIDDEN + ke), (HIDDEN, FFN + ke)]
        attn = 4.0 * case["batch"] * HEADS * HEAD_DIM * case["seq"] * (case["seq"] + 1) / 2
        return {"bytes": 4 * rows * HIDDEN + sum(_packed(n, ke_) for n, ke_ in shapes),
                "flops": attn + sum(_gemm(rows, n, ke_) for n, ke_ in shapes)}
    # every expert that can have a token is read once
    active = min(EXPERTS, rows * TOP_K)
    weights = active * (_packed(2 * FFN, HIDDEN + ke) + _packed(HIDDEN, FFN + ke))
    copies = rows * TOP_K
    return {"bytes": 4 * rows * HIDDEN + weights,
            "flops": _gemm(copies, 2 * FFN, HIDDEN + ke) + _gemm(copies, HIDDEN, FFN + ke)}


def tolerance(case):
    """Codes, scales and statistics are whole numbers or exact maxima.  One GEMM: fp32 sums rounded to bf16 (a
    sum in another order moves an element by one bf16 step now and then).  A block of several quantized GEMMs:
    such a step can move the 4-bit code of a later stage."""
    if case["kind"] in ("calibrate", "pack", "quantize"):
        return "exact"
    if case["kind"] in ("norm_linear", "linear"):
        return {"rel": 2e-3, "max": 2e-2}
    return {"rel": 1e-2}
