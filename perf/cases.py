"""Performance cases of the quantized MoE layer and of the dense GEMMs it is made of: what a program that uses this
framework has it do on one GPU.

A case is a dict of plain values.  Two kinds exist:

  "layer"  one forward pass of DeepseekV3MoE, called as a model calls it (hidden states in, hidden states out), with the
           weights quantized once beforehand
  "gemm"   one quantized linear layer: activation quantizer, then the blockwise GEMM (fp8 or w4a8)

listed() gives the cases, draw() further ones of the same ranges, prepare() a state, run() one pass."""
import math

import torch

from llm_kernels_b200.moe.all2all_moe import DeepseekV3MoE
from llm_kernels_b200.quantization import fp8_kernel, w4a8_kernel
from llm_kernels_b200.workloads import LayerShape, fill_layer_gpu, make_config

# Layer families: hidden size, expert width, experts, experts per token, router groups, groups kept, scoring, scaling.
FAMILIES = {
    "small": (1024, 2048, 8, 2, 1, 1, "softmax", 1.0),         # a small MoE layer
    "dsv3": (7168, 2048, 256, 8, 8, 4, "sigmoid", 2.5),        # DeepSeek-V3 layer, all experts on one GPU
    "dsv3_cut": (7168, 2048, 32, 4, 4, 2, "sigmoid", 2.5),     # one eighth of it: what an expert-parallel rank of 8 holds
    "mixtral": (4096, 14336, 8, 2, 1, 1, "softmax", 1.0),      # few wide experts
}


def _layer(family, method, tokens, skew=0.0, act="silu", shared=0, name=None):
    c = {"kind": "layer", "family": family, "method": method, "tokens": tokens, "skew": skew, "act": act, "shared": shared}
    return c if name is None else dict(c, name=name)


def _gemm(method, m, n, k, name=None):
    c = {"kind": "gemm", "method": method, "m": m, "n": n, "k": k}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # A batch through a small layer: short kernels, so launches and host work count.
        _layer("small", "fp8_block", 512, name="fp8_small_512"),
        # Single-stream decode of a DeepSeek-V3 layer: the weights of eight experts, one row each.
        _layer("dsv3", "fp8_block", 1, name="fp8_decode_1"),
        # Batched decode, a ragged batch: most experts are hit by a few rows.
        _layer("dsv3", "fp8_block", 77, name="fp8_decode_77"),
        # Prefill of 4096 tokens with a Zipf-skewed expert popularity: hot experts with many tiles, some without rows.
        _layer("dsv3", "fp8_block", 4096, skew=1.0, name="fp8_prefill_4096"),
        # A chunk of an odd length on a rank's share of the experts, with a shared expert and GELU.
        _layer("dsv3_cut", "fp8_block", 1001, skew=1.0, act="gelu", shared=1, name="fp8_shared_1001"),
        # Decode of a Mixtral-shape int4 layer with bf16 activations: every expert, about ten rows each.
        _layer("mixtral", "w4a16", 40, name="w4a16_decode_40"),
        # Prefill of the same layer: tensor-core bound.
        _layer("mixtral", "w4a16", 8192, name="w4a16_prefill_8192"),
        # Decode of a DeepSeek-V3 layer with int4 weights and int8 activations.
        _layer("dsv3", "w4a8", 64, name="w4a8_decode_64"),
        # A prefill chunk of it.
        _layer("dsv3", "w4a8", 3000, name="w4a8_prefill_3000"),
        # Quantized linear layers: a decode batch and a prefill batch in fp8, a decode batch with int4 weights.
        _gemm("fp8", 16, 7168, 7168, name="fp8_gemm_16"),
        _gemm("fp8", 4096, 7168, 7168, name="fp8_gemm_4096"),
        _gemm("w4a8", 24, 4096, 7168, name="w4a8_gemm_24"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind and family at random, sizes spread over the logarithm of their range."""
    kind = rng.choice(["small", "fp8", "fp8", "fp8_cut", "w4a16", "w4a8", "gemm_fp8", "gemm_w4a8"])
    skew = rng.choice([0.0, 1.0])
    act = rng.choice(["silu", "silu", "gelu"])
    if kind == "small":
        return _layer("small", "fp8_block", _log_int(rng, 1, 4096), act=act, shared=rng.choice([0, 0, 1]))
    if kind == "fp8":
        return _layer("dsv3", "fp8_block", _log_int(rng, 1, 4096), skew=skew, act=act)
    if kind == "fp8_cut":
        return _layer("dsv3_cut", "fp8_block", _log_int(rng, 1, 4096), skew=skew, act=act, shared=rng.choice([0, 1]))
    if kind == "w4a16":
        return _layer("mixtral", "w4a16", _log_int(rng, 1, 8192), act=act)
    if kind == "w4a8":
        return _layer("dsv3", "w4a8", _log_int(rng, 1, 3000), act=act)
    n, k = 128 * _log_int(rng, 4, 56), 128 * _log_int(rng, 4, 56)
    if kind == "gemm_fp8":
        return _gemm("fp8", _log_int(rng, 1, 4096), n, k)
    return _gemm("w4a8", _log_int(rng, 1, 4096), n, k)


def _shape(case, seed):
    H, I, E, k, g, kept, scoring, scaling = FAMILIES[case["family"]]
    return LayerShape("case", case["tokens"], H, I, E, k, g, kept, scoring, scaling, seed, zipf_bias=case["skew"],
                      method=case["method"])


def _normal(seed, *shape):
    """bf16 values ~N(0,1) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)


def prepare(case, seed):
    """What the program holds before the call: the layer (or the quantized weight) and the activations."""
    if case["kind"] == "gemm":
        w = _normal(2 * seed + 1, case["n"], case["k"]).float().mul_(0.02)
        weight = (fp8_kernel if case["method"] == "fp8" else w4a8_kernel).weight_quant(w)
        return {"gemm": case["method"], "x": _normal(2 * seed, case["m"], case["k"]), "weight": weight}
    shape = _shape(case, seed)
    cfg = make_config(shape)
    cfg.hidden_act, cfg.n_shared_experts = case["act"], case["shared"]
    layer = DeepseekV3MoE(cfg).eval()
    fill_layer_gpu(layer, shape)
    if case["shared"]:
        wide = shape.inter * case["shared"]
        w = [_normal(2 * seed + 3 + i, *s).mul_(0.02) for i, s in
             enumerate(((wide, shape.hidden), (wide, shape.hidden), (shape.hidden, wide)))]
        layer.load_shared_experts(*w)
    return {"layer": layer, "x": _normal(2 * seed, 1, case["tokens"], shape.hidden)}


def run(state):
    if "layer" in state:
        return state["layer"](state["x"])
    if state["gemm"] == "fp8":
        q, s = fp8_kernel.act_quant(state["x"])
        return fp8_kernel.fp8_gemm(q, s, *state["weight"], out_dtype=torch.bfloat16)
    q, s = w4a8_kernel.act_quant(state["x"])
    return w4a8_kernel.w4a8_gemm(q, s, *state["weight"], out_dtype=torch.bfloat16)


def _active_experts(case):
    """Experts that receive at least one row, in the mean over the routers of such a layer: the selection restated on
    random logits of the layer's distribution."""
    H, _, E, k, groups, kept, scoring, _ = FAMILIES[case["family"]]
    g = torch.Generator().manual_seed(1)
    T = case["tokens"]
    trials = max(1, 64 // T)
    logits = torch.randn(trials * T, E, generator=g) * 0.02 * math.sqrt(H)
    score = logits.sigmoid() if scoring == "sigmoid" else logits.softmax(-1)
    if case["skew"]:
        score = score + case["skew"] * 0.08 * 1.1 * (math.log(E) - torch.arange(1, E + 1).log())[torch.randperm(E, generator=g)]
    best = score.view(-1, groups, E // groups).topk(min(2, E // groups), dim=-1)[0].sum(-1)
    keep = torch.zeros_like(best).scatter_(1, best.topk(kept, dim=-1)[1], 1.0).repeat_interleave(E // groups, 1)
    idx = (score * keep).topk(k, dim=-1)[1].view(trials, T * k)
    return sum(len(set(row.tolist())) for row in idx) / trials


# Bytes of one weight with its share of the scales (and zero points).
_WEIGHT_BYTES = {"fp8_block": 1 + 4 / 16384, "w4a16": 0.5 + 4 / 128, "w4a8": 0.5 + 2 / 128 + 4 / 16384,
                 "fp8": 1 + 4 / 16384}


def work(case):
    """Each input read once (the weights of the experts that receive rows), each output written once."""
    if case["kind"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * m * k + 2 * m * n + n * k * _WEIGHT_BYTES[case["method"]], "flops": 2.0 * m * n * k}
    H, I, E, k = FAMILIES[case["family"]][:4]
    T, wide = case["tokens"], FAMILIES[case["family"]][1] * case["shared"]
    return {"bytes": 4 * T * H + 4 * E * H + _active_experts(case) * 3 * H * I * _WEIGHT_BYTES[case["method"]] + 6 * H * wide,
            "flops": 6.0 * H * I * T * k + 2.0 * T * H * E + 6.0 * H * wide * T}


def tolerance(case):
    """bf16 results.  The fp8 and w4a8 layers round their activations to 8 bits twice, where a last-bit difference of a
    sum can move a value to its neighbour; the GEMMs and the w4a16 layer only round sums to bf16."""
    if case["kind"] == "layer" and case["method"] != "w4a16":
        return {"rel": 1e-2}
    return {"rel": 3e-3}
