"""What this framework is timed on: weight-only-quantised linears as a language model's inference calls
them, through the public entry points (`ipex_b200.llm.optimize`, the fusion modules it leaves behind, the
module forward and the MoE operator).

A case is one decoder layer's linears (`op` "layer"), a single linear ("linear") or a mixture-of-experts
layer ("moe") of a given architecture, weight recipe and token count.  Layer sizes are those of the
Llama-3-8B, Llama-3-70B and Mixtral-8x7B architectures this repository's benchmark runs; weights are
N(0, 0.02), activations N(0, 1) bf16, as its configurations state.  Attention, norms and the router's
matrix product are not weight-only-quantised linears and stay outside.

Decode cases are replayed from a CUDA graph, as a serving loop does it (`bench.py`, `bench_stack.py`);
everything else is called eagerly.
"""
import math
import os
import sys

import torch
from torch import nn

sys.path.insert(0, os.path.join(os.getcwd(), "intel-extension-for-pytorch_b200"))
import ipex_b200  # noqa: E402
from ipex_b200 import quantization as Q  # noqa: E402
from ipex_b200.nn.modules import WeightOnlyQuantizedLinear  # noqa: E402
from ipex_b200.transformers.fusions.linear_fusion import _IPEXlinearAdd, _IPEXlinearSiluMul  # noqa: E402

# name -> (weight dtype, low-precision compute mode, activation quantisation mode)
RECIPES = {
    # INT4 checkpoints with bf16 compute: the recipe of the headline benchmark
    "int4": (Q.WoqWeightDtype.INT4, Q.WoqLowpMode.BF16, Q.WoqActQuantMode.NONE),
    # INT8 weights and compute, one activation scale per token
    "int8_int8": (Q.WoqWeightDtype.INT8, Q.WoqLowpMode.INT8, Q.WoqActQuantMode.PER_BATCH_SYM),
    # INT4 weights, INT8 compute with the qconfig factory's default activation mode (per token and K block)
    "int4_int8": (Q.WoqWeightDtype.INT4, Q.WoqLowpMode.INT8, Q.WoqActQuantMode.PER_BATCH_IC_BLOCK_SYM),
    # get_weight_only_quant_qconfig_mapping() with no arguments: asymmetric per-channel INT8, activation dtype kept
    "default": (Q.WoqWeightDtype.INT8, Q.WoqLowpMode.NONE, Q.WoqActQuantMode.NONE),
    # NormalFloat4 weights, activation dtype kept
    "nf4": (Q.WoqWeightDtype.NF4, Q.WoqLowpMode.NONE, Q.WoqActQuantMode.NONE),
}

# hidden size, key/value projection rows, feed-forward size
LLAMA_8B = dict(hidden=4096, kv=1024, ffn=14336)
LLAMA_70B = dict(hidden=8192, kv=1024, ffn=28672)


def listed():
    return [
        # the smallest call: one attention output projection for one token, called eagerly (latency)
        dict(name="int4_linear_1", op="linear", recipe="int4", n=4096, k=4096, group=128, tokens=1, graph=False),
        # one user's decode step of an 8B model (two layers: a step's weights do not stay in L2)
        dict(name="int4_8b_decode_1", op="layer", recipe="int4", group=128, tokens=1, layers=2, graph=True, **LLAMA_8B),
        # batched serving: one token for each of 32 sequences
        dict(name="int4_8b_decode_32", op="layer", recipe="int4", group=128, tokens=32, layers=2, graph=True, **LLAMA_8B),
        # one user's decode step of a 70B model on one GPU: the headline benchmark's layer
        dict(name="int4_70b_decode_1", op="layer", recipe="int4", group=128, tokens=1, layers=1, graph=True, **LLAMA_70B),
        # large-batch decode of a 70B model
        dict(name="int4_70b_decode_128", op="layer", recipe="int4", group=128, tokens=128, layers=1, graph=True,
             **LLAMA_70B),
        # prefill of one prompt whose length is no multiple of anything
        dict(name="int4_8b_prefill_1000", op="layer", recipe="int4", group=128, tokens=1000, layers=1, graph=False,
             **LLAMA_8B),
        # prefill of a batch of long prompts on a 70B model: the largest call
        dict(name="int4_70b_prefill_4096", op="layer", recipe="int4", group=128, tokens=4096, layers=1, graph=False,
             **LLAMA_70B),
        # INT8 compute: decode for a few sequences, and prefill
        dict(name="int8_8b_decode_8", op="layer", recipe="int8_int8", group=-1, tokens=8, layers=2, graph=True, **LLAMA_8B),
        dict(name="int8_8b_prefill_512", op="layer", recipe="int8_int8", group=-1, tokens=512, layers=1, graph=False,
             **LLAMA_8B),
        # INT4 weights with INT8 compute at a batch between decode and prefill
        dict(name="int4_int8_8b_64", op="layer", recipe="int4_int8", group=128, tokens=64, layers=1, graph=False, **LLAMA_8B),
        # the qconfig factory's defaults, decode for a few sequences
        dict(name="default_8b_decode_8", op="layer", recipe="default", group=-1, tokens=8, layers=1, graph=True, **LLAMA_8B),
        # Mixtral's expert layer for a mid-sized batch: 8 experts, 2 per token
        dict(name="moe_256", op="moe", recipe="int4", group=128, tokens=256, experts=8, top_k=2, hidden=4096, ffn=14336),
    ]


def _log(rng, lo, hi, step=1):
    """A whole number between lo and hi, spread over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(["decode", "decode", "batch", "batch", "prefill", "prefill", "int8", "int8", "int4_int8",
                       "default", "nf4", "moe", "linear"])
    if kind == "moe":
        return dict(op="moe", recipe="int4", group=128, tokens=_log(rng, 1, 4096), experts=rng.choice([4, 8]), top_k=2,
                    hidden=128 * rng.randint(8, 40), ffn=128 * rng.randint(16, 112))
    if kind == "linear":
        # any number of output rows (classification heads, adapters, sharded vocabularies)
        return dict(op="linear", recipe="int4", n=_log(rng, 256, 32768), k=64 * rng.randint(16, 200),
                    group=rng.choice([64, 128]), tokens=_log(rng, 1, 2048), graph=False)
    hidden = 128 * rng.randint(8, 64)
    arch = dict(hidden=hidden, kv=128 * rng.randint(1, max(1, hidden // 512)), ffn=128 * rng.randint(16, 224))
    if kind == "decode":
        return dict(op="layer", recipe="int4", group=rng.choice([64, 128, 128, -1]), tokens=_log(rng, 1, 16),
                    layers=rng.choice([1, 2]), graph=True, **arch)
    if kind == "batch":
        return dict(op="layer", recipe="int4", group=rng.choice([64, 128, 128, -1]), tokens=_log(rng, 17, 256),
                    layers=1, graph=rng.random() < 0.5, **arch)
    if kind == "prefill":
        return dict(op="layer", recipe="int4", group=rng.choice([64, 128, 128, -1]), tokens=_log(rng, 257, 4096),
                    layers=1, graph=False, **arch)
    if kind == "int8":
        return dict(op="layer", recipe="int8_int8", group=-1, tokens=_log(rng, 1, 2048), layers=1,
                    graph=rng.random() < 0.5, **arch)
    if kind == "int4_int8":
        return dict(op="layer", recipe="int4_int8", group=128, tokens=_log(rng, 1, 512), layers=1, graph=False, **arch)
    arch["ffn"] = min(arch["ffn"], 14336)
    return dict(op="layer", recipe=kind, group=-1 if kind == "default" else rng.choice([64, 128]),
                tokens=_log(rng, 1, 256), layers=1, graph=False, **arch)


class _Attention(nn.Module):
    def __init__(self, hidden, kv, make):
        super().__init__()
        self.q_proj, self.k_proj, self.v_proj = make(hidden, hidden), make(kv, hidden), make(kv, hidden)
        self.o_proj = make(hidden, hidden)


class _Mlp(nn.Module):
    def __init__(self, hidden, ffn, make):
        super().__init__()
        self.gate_proj, self.up_proj, self.down_proj = make(ffn, hidden), make(ffn, hidden), make(hidden, ffn)
        self.act_fn = nn.SiLU()


class _Layer(nn.Module):
    """The linears of a Llama-style decoder layer under the names `llm.optimize` looks for."""

    def __init__(self, hidden, kv, ffn, make):
        super().__init__()
        self.self_attn = _Attention(hidden, kv, make)
        self.mlp = _Mlp(hidden, ffn, make)


def _maker(gen):
    def make(n, k):
        lin = nn.Linear(k, n, bias=False, device="cuda", dtype=torch.bfloat16)
        with torch.no_grad():
            lin.weight.copy_(torch.randn(n, k, generator=gen, device="cuda", dtype=torch.bfloat16).mul_(0.02))
        return lin

    return make


def _qmap(case):
    dtype, lowp, act = RECIPES[case["recipe"]]
    return Q.get_weight_only_quant_qconfig_mapping(weight_dtype=dtype, lowp_mode=lowp, act_quant_mode=act,
                                                   group_size=case["group"])


def _quantised(case, make, n, k):
    lin = make(n, k)
    lin.qconfig = _qmap(case).global_qconfig
    return WeightOnlyQuantizedLinear.from_float(lin)


def _layer_pass(layers, acts):
    outs = []
    for layer, a in zip(layers, acts):
        qkv = layer.self_attn.qkv_concat.concat(a["x"])
        h = layer.mha_linear_add(a["attn"], a["residual"])
        act = layer.gate_up(a["h"])
        outs += [qkv, h, act, layer.mlp_linear_add(act, a["residual"])]
    return outs


def prepare(case, seed):
    """Quantised and packed modules, activations on the device and, for a decode loop, its CUDA graph."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    make = _maker(gen)
    t = case["tokens"]

    def acts(width):
        return torch.randn(t, width, generator=gen, device="cuda", dtype=torch.bfloat16)

    if case["op"] == "moe":
        hidden, ffn = case["hidden"], case["ffn"]
        experts = [[_quantised(case, make, n, k) for n, k in ((ffn, hidden), (ffn, hidden), (hidden, ffn))]
                   for _ in range(case["experts"])]
        for mods in experts:
            for m in mods:
                m.weight = None  # the plain copy the module keeps for queries
        # a softmax router's choice: top-k experts and their renormalised probabilities
        p = torch.softmax(torch.randn(t, case["experts"], generator=gen, device="cuda"), -1)
        w, ids = torch.topk(p, case["top_k"], -1)
        ctxs = [[mods[i]._op_context for mods in experts] for i in range(3)]
        return dict(op="moe", x=acts(hidden), ids=ids, w=(w / w.sum(-1, keepdim=True)).to(torch.bfloat16), ctxs=ctxs)
    if case["op"] == "linear":
        state = dict(op="linear", mod=_quantised(case, make, case["n"], case["k"]), x=acts(case["k"]))
        state["mod"].weight = None
        return state

    layers, inputs = [], []
    for _ in range(case["layers"]):
        layer = _Layer(case["hidden"], case["kv"], case["ffn"], make)
        layer = ipex_b200.llm.optimize(layer, quantization_config=_qmap(case), inplace=True)
        mlp = layer.mlp
        layer.gate_up = mlp.gate_up_fused if hasattr(mlp, "gate_up_fused") else _IPEXlinearSiluMul(mlp.gate_proj, mlp.up_proj)
        for m in layer.modules():
            if isinstance(m, WeightOnlyQuantizedLinear):
                m.weight = None
        layers.append(layer)
        inputs.append(dict(x=acts(case["hidden"]), attn=acts(case["hidden"]), residual=acts(case["hidden"]),
                           h=acts(case["hidden"])))
    state = dict(op="layer", layers=layers, acts=inputs)
    if case["graph"]:
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _layer_pass(layers, inputs)
        torch.cuda.current_stream().wait_stream(stream)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"], stream=stream):
            state["outs"] = _layer_pass(layers, inputs)
    return state


def run(state):
    if state["op"] == "moe":
        return torch.ops.torch_ipex.deepseek_moe_woq(state["x"], state["ids"], *state["ctxs"], state["w"], False)
    if state["op"] == "linear":
        return state["mod"](state["x"])
    if "graph" in state:
        state["graph"].replay()
        return state["outs"]
    return _layer_pass(state["layers"], state["acts"])


def _linears(case):
    """(output rows, K, tokens, output width, extra operands) of every linear of a pass."""
    t = case["tokens"]
    if case["op"] == "linear":
        return [(case["n"], case["k"], t, case["n"], 0)]
    hidden, ffn = case["hidden"], case["ffn"]
    if case["op"] == "moe":
        pairs = t * case["top_k"]
        used = min(case["experts"], pairs)  # experts that are read, when there are fewer tokens than experts
        return [(2 * ffn * used, hidden, pairs / used, ffn * used, 0), (hidden * used, ffn, pairs / used, hidden * used, 0)]
    return [(hidden + 2 * case["kv"], hidden, t, hidden + 2 * case["kv"], 0), (hidden, hidden, t, hidden, 1),
            (2 * ffn, hidden, t, ffn, 0), (hidden, ffn, t, hidden, 1)] * case["layers"]


def work(case):
    """Packed weights with their scales and zero points, activations, extra operands and results, once each."""
    dtype = RECIPES[case["recipe"]][0]
    total, flops = 0, 0
    for n, k, t, width, extra in _linears(case):
        weight = n * k if dtype == Q.WoqWeightDtype.INT8 else n * k // 2
        groups = k / case["group"] if case["group"] > 0 else 1
        total += weight + 3 * n * groups
        if case["op"] != "moe":
            total += 2 * k * t + 2 * width * t * (1 + extra)
        flops += 2 * n * k * t
    if case["op"] == "moe":
        total += 2 * 2 * case["hidden"] * case["tokens"]
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Four times what sums in another order show.  Against the same linears summed in 64 bits (each result rounded
    to bf16 once, as here), one linear differs by 1e-4 .. 2e-4 in the 2-norm and the chain gate/up, silu*mul, down
    projection, residual by 3e-4 .. 9e-4: nearly equal sums that round to neighbouring bf16 values.  An INT8 chain
    quantises such values again, and the MoE layer adds its experts' shares in bf16 (2e-3 against 64-bit sums)."""
    return {"rel": 8e-3 if case["op"] == "moe" or case["recipe"] in ("int8_int8", "int4_int8") else 3.5e-3}
