"""The work that a serving program has this package do, as a list of cases and a way to draw more of the same kind.

Four kinds of case, each one pass through the package's public entry points:

``linear``       one quantised linear layer on its own: what a caller of a single projection waits for.
``projections``  the four linears of a decoder layer (qkv, o_proj, gate_up, down), each on an input of its own, as they
                 run in a model whose norms, attention and activation belong to the caller.
``decoder``      a stack of W8A8 decoder layers without their attention: RMSNorm -> e4m3 codes -> qkv -> o_proj ->
                 RMSNorm -> e4m3 codes -> fused MLP, with the residual stream updated in place.  ``graph`` replays the
                 stack from a CUDA graph on static buffers, as a decode loop does; without it the layers are called
                 one after the other, as for a prompt or in an eager loop.
``moe``          router, grouped expert FFN and combine of one mixture-of-experts block.

Shapes are those of the 3B- and 7B-sized dense models (hidden 2048 / 3584, intermediate 11008 / 18944) and of the
60-expert block (hidden 2048, expert intermediate 1408, top 4) of this repository's benchmark.  Weights are N(0, 0.02)
in e4m3 with one scale per output channel, activations N(0, 1), activation scales amax / 448 of a calibration draw.
"""
from __future__ import annotations

import importlib
import math

import torch

fp8 = importlib.import_module("nano-vllm-moe_b200")
export = importlib.import_module("nano-vllm-moe_b200.quantization.export")
moe = importlib.import_module("nano-vllm-moe_b200.executor.moe")

SCHEMES = {"w8a8": "fp8_w8a8_static", "w8a16": "fp8_w8a16"}
HEAD = 128
WEIGHT_STD = 0.02


def _linear(name, scheme, rows, k, n, bias):
    return {"name": name, "kind": "linear", "scheme": scheme, "rows": rows, "k": k, "n": n, "bias": bias}


def _projections(name, scheme, rows, hidden=3584, heads=28, kv_heads=4, inter=18944):
    return {"name": name, "kind": "projections", "scheme": scheme, "rows": rows, "hidden": hidden, "heads": heads,
            "kv_heads": kv_heads, "inter": inter}


def _decoder(name, rows, layers, graph, hidden=3584, heads=28, kv_heads=4, inter=18944):
    return {"name": name, "kind": "decoder", "scheme": "w8a8", "rows": rows, "layers": layers, "graph": graph,
            "hidden": hidden, "heads": heads, "kv_heads": kv_heads, "inter": inter}


def _moe(name, rows, hidden=2048, experts=60, inter=1408, top_k=4):
    return {"name": name, "kind": "moe", "scheme": "w8a8", "rows": rows, "hidden": hidden, "experts": experts,
            "inter": inter, "top_k": top_k}


def listed():
    return [
        # one token through the smallest projection of the 3B model: launch count and host time are everything
        _linear("linear_w8a8_r1", "w8a8", 1, 2048, 2048, True),
        # a small decode batch through the 3B gate_up half, weights widened on the fly
        _linear("linear_w8a16_r16", "w8a16", 16, 2048, 11008, False),
        # a short prompt through the 3B down projection: long K, few output tiles
        _linear("linear_w8a8_r256", "w8a8", 256, 11008, 2048, True),
        # weight-only serving of a few concurrent users, 7B layer
        _projections("projections_w8a16_r4", "w8a16", 4),
        # weight-only, a ragged mid-sized batch (chunked prefill beside decode), 7B layer
        _projections("projections_w8a16_r200", "w8a16", 200),
        # weight-only prefill, 7B layer
        _projections("projections_w8a16_r4096", "w8a16", 4096),
        # the largest: a full W8A8 prefill batch, 7B layer
        _projections("projections_w8a8_r16384", "w8a8", 16384),
        # single-user decode in an eager loop, four 7B layers
        _decoder("decoder_r1", 1, 4, False),
        # batched decode replayed from a CUDA graph, four 7B layers
        _decoder("decoder_graph_r64", 64, 4, True),
        # a ragged prompt through two 7B layers
        _decoder("decoder_r1031", 1031, 2, False),
        # decode batch through the expert block: every expert's weights are touched by a few rows
        _moe("moe_r64", 64),
        # prefill through the expert block
        _moe("moe_r4096", 4096),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _dense_sizes(rng):
    """Hidden size, heads and intermediate size of a dense model between the small and the 7B one."""
    kv_heads = rng.choice([2, 4])
    heads = kv_heads * rng.randint(8 // kv_heads, 28 // kv_heads)
    hidden = heads * HEAD
    inter = 128 * min(148, max(16, int(heads * rng.uniform(2.5, 5.5))))
    return {"hidden": hidden, "heads": heads, "kv_heads": kv_heads, "inter": inter}


def draw(rng):
    kind = rng.choice(["linear", "projections", "decoder", "moe"])
    if kind == "linear":
        # rows over the whole range; widths down to a tensor-parallel shard, seldom a multiple of the tiles
        scheme = rng.choice(list(SCHEMES))
        case = _linear("", scheme, _log_int(rng, 1, 8192 if scheme == "w8a8" else 4096), 16 * _log_int(rng, 28, 1184),
                       8 * _log_int(rng, 64, 4736), rng.random() < 0.5)
    elif kind == "projections":
        scheme = rng.choice(list(SCHEMES))
        case = _projections("", scheme, _log_int(rng, 1, 16384 if scheme == "w8a8" else 4096), **_dense_sizes(rng))
    elif kind == "decoder":
        graph = rng.random() < 0.5
        # a decode loop captures its graphs up to some batch size; eager passes are single users up to whole prompts
        case = _decoder("", _log_int(rng, 1, 128 if graph else 2048), rng.randint(2, 4), graph, **_dense_sizes(rng))
    else:
        case = _moe("", _log_int(rng, 1, 4096), 128 * rng.randint(8, 16), rng.randint(8, 64), 16 * rng.randint(32, 88),
                    rng.choice([2, 4, 8]))
    del case["name"]
    return case


# ---- preparation ---------------------------------------------------------------------------------------------------

class _State:
    """What a serving program keeps: layers, weights, input and output buffers."""


def _randn(gen, *shape, std=1.0):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32).mul_(std).to(torch.bfloat16)


def _static_scale(sample):
    return sample.abs().amax().float() / 448.0


def _fill(layer, gen, k, n, input_scale, bias):
    """Load random checkpoint tensors into a layer through its weight loaders and make it ready."""
    codes, scale = export.quantize_weight(_randn(gen, n, k, std=WEIGHT_STD))
    layer.qweight.weight_loader(layer.qweight, codes)
    layer.weight_scale.weight_loader(layer.weight_scale, scale)
    if input_scale is not None:
        layer.input_scale.weight_loader(layer.input_scale, input_scale)
    if bias:
        layer.bias.data = _randn(gen, n, std=0.01)
    fp8.process_weights_after_loading(layer)
    return layer


def _method(scheme):
    return fp8.Fp8Config(SCHEMES[scheme]).get_quant_method(None)


def _layer_linears(case, gen, scales):
    """qkv, o_proj, gate_up and down of one decoder layer; ``scales``: their input scales, or None for W8A16."""
    scheme, hidden, inter = case["scheme"], case["hidden"], case["inter"]
    heads, kv = case["heads"], case["kv_heads"]
    with torch.device("cuda"):
        layers = [
            fp8.QKVParallelLinear(hidden, HEAD, heads, kv, bias=True, quant_method=_method(scheme)),
            fp8.RowParallelLinear(heads * HEAD, hidden, quant_method=_method(scheme)),
            fp8.MergedColumnParallelLinear(hidden, [inter, inter], quant_method=_method(scheme)),
            fp8.RowParallelLinear(inter, hidden, quant_method=_method(scheme)),
        ]
    widths = _layer_widths(case)
    return [_fill(lay, gen, k, n, scales[i] if scheme == "w8a8" else None, i == 0)
            for i, (lay, (k, n)) in enumerate(zip(layers, widths))]


def _layer_widths(case):
    qkv = (case["heads"] + 2 * case["kv_heads"]) * HEAD
    return [(case["hidden"], qkv), (case["heads"] * HEAD, case["hidden"]), (case["hidden"], 2 * case["inter"]),
            (case["inter"], case["hidden"])]


def _prepare_linear(case, gen, s):
    k, n = case["k"], case["n"]
    s.x = _randn(gen, case["rows"], k)
    scale = _static_scale(_randn(gen, 512, k)) if case["scheme"] == "w8a8" else None
    with torch.device("cuda"):
        layer = fp8.ColumnParallelLinear(k, n, bias=case["bias"], quant_method=_method(case["scheme"]))
    s.layer = _fill(layer, gen, k, n, scale, case["bias"])


def _prepare_projections(case, gen, s):
    scale = _static_scale(_randn(gen, 512, case["hidden"]))
    s.linears = _layer_linears(case, gen, [scale] * 4)
    s.xs = [_randn(gen, case["rows"], k) for k, _ in _layer_widths(case)]


def _prepare_decoder(case, gen, s):
    rows, hidden = case["rows"], case["hidden"]
    std = WEIGHT_STD * math.sqrt(hidden)                    # of a projection of a normalised row
    normed = _static_scale(_randn(gen, 512, hidden))
    attn = _static_scale(_randn(gen, 512, hidden, std=std))
    gate, up = _randn(gen, 512, hidden, std=std), _randn(gen, 512, hidden, std=std)
    act = _static_scale(torch.nn.functional.silu(gate) * up)
    s.layers = []
    for _ in range(case["layers"]):
        qkv, o_proj, gate_up, down = _layer_linears(case, gen, [normed, attn, normed, act])
        norms = [fp8.RMSNorm(hidden).to(device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        for norm in norms:
            norm.weight.data.add_(_randn(gen, hidden, std=0.1))
        s.layers.append((norms[0], qkv, o_proj, norms[1], gate_up, fp8.FusedFp8MLP(gate_up, down, release_unfused=True)))
    s.q_width = case["heads"] * HEAD
    s.x = _randn(gen, rows, hidden)
    s.graph = None
    if case["graph"]:
        s.residual = torch.empty_like(s.x)
        s.residual.copy_(s.x)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _decoder_pass(s, s.residual)                    # scratch of this stream exists before the capture
        stream.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph, stream=stream):
            s.out = _decoder_pass(s, s.residual)


def _decoder_pass(s, residual):
    """The stack on ``residual`` (updated in place); attention is replaced by the q columns of the qkv result."""
    hidden = None
    for first, qkv, o_proj, second, gate_up, mlp in s.layers:
        if hidden is None:
            codes, _ = first.forward_quant(residual, qkv.input_scale)
        else:
            codes, residual = first.forward_quant(hidden, qkv.input_scale, residual)
        hidden = o_proj(qkv(codes)[:, :s.q_width])
        codes, residual = second.forward_quant(hidden, gate_up.input_scale, residual)
        hidden = mlp(codes)
    return hidden, residual


def _prepare_moe(case, gen, s):
    rows, hidden, experts, inter = case["rows"], case["hidden"], case["experts"], case["inter"]
    w13, w13_scale = export.quantize_weight(_randn(gen, experts * 2 * inter, hidden, std=WEIGHT_STD))
    w2, w2_scale = export.quantize_weight(_randn(gen, experts * hidden, inter, std=WEIGHT_STD))
    std = WEIGHT_STD * math.sqrt(hidden)
    act = torch.nn.functional.silu(_randn(gen, 512, inter, std=std)) * _randn(gen, 512, inter, std=std)
    s.weights = moe.Fp8ExpertWeights.from_checkpoint_layout(
        w13.view(experts, 2 * inter, hidden), w13_scale.view(experts, 2 * inter), _static_scale(_randn(gen, 512, hidden)),
        w2.view(experts, hidden, inter), w2_scale.view(experts, hidden), _static_scale(act))
    cfg = moe.make_moe_parallel_config(tp_group=None, ep_group=None, global_num_experts=experts, intermediate_size=inter)
    s.router = moe.SoftmaxTopKRouter(case["top_k"], renormalize=False)
    s.block = moe.MoEKernel(prepare_finalize=moe.NoEPPrepareFinalize(cfg), experts=moe.Fp8Experts(), parallel_config=cfg)
    s.x = _randn(gen, rows, hidden)
    s.logits = _randn(gen, rows, experts)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = _State()
    s.kind = case["kind"]
    {"linear": _prepare_linear, "projections": _prepare_projections, "decoder": _prepare_decoder,
     "moe": _prepare_moe}[s.kind](case, gen, s)
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------

@torch.inference_mode()
def run(s):
    if s.kind == "linear":
        return s.layer(s.x)
    if s.kind == "projections":
        return [layer(x) for layer, x in zip(s.linears, s.xs)]
    if s.kind == "moe":
        weights, ids = s.router.select_experts(s.x, s.logits)
        return s.block(s.x, weights, ids, s.weights, model_dtype=torch.bfloat16)
    if s.graph is None:
        return _decoder_pass(s, s.x.clone())
    s.residual.copy_(s.x)                                   # the new tokens' rows into the static buffer
    s.graph.replay()
    return s.out


def work(case):
    rows = case["rows"]
    if case["kind"] == "linear":
        k, n = case["k"], case["n"]
        return {"bytes": 2 * rows * k + k * n + 4 * n + (2 * n if case["bias"] else 0) + 2 * rows * n,
                "flops": 2 * rows * k * n}
    if case["kind"] == "projections":
        return {"bytes": sum(2 * rows * k + k * n + 4 * n + 2 * rows * n for k, n in _layer_widths(case)),
                "flops": sum(2 * rows * k * n for k, n in _layer_widths(case))}
    if case["kind"] == "decoder":
        # the weights once, the input rows, and the two results
        weights = sum(k * n + 4 * n for k, n in _layer_widths(case))
        return {"bytes": case["layers"] * weights + 6 * rows * case["hidden"],
                "flops": case["layers"] * sum(2 * rows * k * n for k, n in _layer_widths(case))}
    # every expert that an evenly spread routing reaches, the token rows in and out, the logits
    hidden, inter, routed = case["hidden"], case["inter"], rows * case["top_k"]
    reached = case["experts"] * (1.0 - (1.0 - case["top_k"] / case["experts"]) ** rows)
    return {"bytes": int(reached * (3 * hidden * inter + 4 * (2 * inter + hidden))) + 4 * rows * hidden + 2 * rows * case["experts"],
            "flops": routed * 6 * hidden * inter}


def tolerance(case):
    # bf16 results of fp32 sums: another order of the same sums moves a result by one bf16 step at most
    if case["kind"] in ("linear", "projections"):
        return {"rel": 5e-3, "max": 3e-2}
    # an e4m3 code between two linears may move by one step (1/16 of the value) where a sum moved
    return {"rel": 1e-2, "max": 0.3} if case["kind"] == "moe" else {"rel": 2e-2, "max": 0.5}
