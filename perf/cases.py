"""Performance cases of the block-FP8 path: the calls a serving program makes, from one decode token to a full prefill.

Four operations, each through its public entry points:

* ``linear``: ``Fp8LinearMethod.apply`` on a loaded layer (quantise the activations, block-scaled GEMM, optional bias),
  on a checkpoint with fp32 weight scales or one with power-of-two (UE8M0) scales;
* ``quant``: ``sglang_per_token_group_quant_fp8`` by itself, in the scale layouts the callers ask for;
* ``moe``: router (softmax top-k or the sigmoid group-limited gate) plus the fused expert MLP, on either checkpoint;
* ``masked``: the expert MLP in the masked per-expert layout a low-latency dispatcher fills, into buffers the caller
  keeps.

Inputs follow the repository's benchmark: activations ~N(0, 1) with 1 % of the entries x50 (rows scaled log-uniformly in
[1e-2, 1e2] for ``quant``), weights ~N(0, 0.02) in 128x128 blocks, router logits ~N(0, 1).
"""

import math

import torch

from sglang_b200.layers.deep_gemm_wrapper import grouped_gemm_nt_f8f8bf16_masked
from sglang_b200.layers.moe import (MoeRunnerConfig, StandardTopKOutput, fused_experts,
                                    fused_experts_block_fp8_ue8m0)
from sglang_b200.layers.moe.topk import biased_grouped_topk, fused_topk
from sglang_b200.layers.quantization.fp8 import Fp8Config, Fp8LinearMethod
from sglang_b200.layers.quantization.fp8_kernel import pack_ue8m0_scales, sglang_per_token_group_quant_fp8
from sglang_b200.layers.quantization.fp8_utils import block_quant_weight_fp8, per_block_cast_to_fp8

DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}

# (N, K) of the projections: the five DeepSeek-V3 layers, the four Llama-3-70B layers, and generic widths
LINEAR_SHAPES = [(24576, 1536), (576, 7168), (7168, 16384), (36864, 7168), (7168, 18432),
                 (10240, 8192), (8192, 8192), (57344, 8192), (8192, 28672),
                 (4096, 4096), (1536, 7168), (2112, 7168), (3072, 1536), (5120, 2560), (1000, 1024)]
# (experts, hidden, moe_intermediate, topk): the DeepSeek-V3 layer and generic layers, one of them few and wide
MOE_SHAPES = [(256, 7168, 2048, 8), (256, 7168, 256, 8), (128, 4096, 1536, 8), (64, 2048, 1408, 6), (8, 4096, 14336, 2)]
LARGEST_FLOPS = 2 * 8192 * 36864 * 7168


def _linear(m, n, k, checkpoint="fp32", dtype="bfloat16", bias=False):
    return {"op": "linear", "m": m, "n": n, "k": k, "checkpoint": checkpoint, "dtype": dtype, "bias": bias}


def _quant(m, k, layout="col_tma", dtype="bfloat16", silu=False):
    return {"op": "quant", "m": m, "k": k, "layout": layout, "dtype": dtype, "silu": silu}


def _moe(m, experts, hidden, inter, topk, checkpoint="fp32"):
    return {"op": "moe", "m": m, "experts": experts, "hidden": hidden, "inter": inter, "topk": topk,
            "checkpoint": checkpoint}


def _masked(experts, max_m, expected_m, hidden, inter):
    return {"op": "masked", "experts": experts, "max_m": max_m, "expected_m": expected_m, "hidden": hidden,
            "inter": inter}


def listed():
    cases = [
        # one decode token through the smallest projection (kv_a): latency, launches and host time only
        ("linear_m1_kv_a", _linear(1, 576, 7168)),
        # an ordinary decode batch through the attention output projection: weight streaming
        ("linear_m16_o_proj", _linear(16, 7168, 16384)),
        # a large decode batch on a UE8M0 checkpoint through the widest projection
        ("linear_m48_gate_up_ue8m0", _linear(48, 36864, 7168, "ue8m0")),
        # a ragged mixed batch (decode rows plus a prompt's tail), fp16 activations and a QKV bias
        ("linear_m113_qkv_f16_bias", _linear(113, 10240, 8192, dtype="float16", bias=True)),
        # a ragged prefill chunk through a short-K projection (q_b)
        ("linear_m777_q_b", _linear(777, 24576, 1536)),
        # prefill on a UE8M0 checkpoint through a long-K projection (down_proj)
        ("linear_m4096_down_ue8m0", _linear(4096, 7168, 18432, "ue8m0")),
        # the largest prefill batch through the widest projection: the largest listed GEMM
        ("linear_m8192_gate_up", _linear(8192, 36864, 7168)),
        # the activation quantiser alone at prefill size
        ("quant_m16384", _quant(16384, 7168)),
        # an ordinary decode batch through a full expert layer, router included
        ("moe_m16", _moe(16, 256, 7168, 2048, 8)),
        # a ragged prompt through the same layer on a UE8M0 checkpoint, group-limited sigmoid gate
        ("moe_m1021_ue8m0", _moe(1021, 256, 7168, 2048, 8, "ue8m0")),
        # prefill through the expert layer
        ("moe_m4096", _moe(4096, 256, 7168, 2048, 8)),
        # decode on one expert-parallel rank of eight: 32 local experts, the dispatcher's masked layout
        ("masked_e32_rows24", _masked(32, 128, 24, 7168, 2048)),
    ]
    return [dict(c, name=name) for name, c in cases]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        op = rng.choices(["linear", "quant", "moe", "masked"], [7, 1.5, 3, 1])[0]
        if op == "linear":
            n, k = rng.choice(LINEAR_SHAPES)
            case = _linear(_log_uniform(rng, 1, 8192), n, k, rng.choice(["fp32", "fp32", "ue8m0"]),
                           rng.choice(["bfloat16", "bfloat16", "bfloat16", "float16"]), rng.random() < 0.15)
        elif op == "quant":
            case = _quant(_log_uniform(rng, 1, 16384), rng.choice([1536, 2048, 4096, 7168]),
                          rng.choice(["row", "col", "col_tma", "ue8m0"]),
                          rng.choice(["bfloat16", "bfloat16", "float16"]), rng.random() < 0.3)
        elif op == "moe":
            e, h, i, topk = rng.choice(MOE_SHAPES)
            checkpoint = rng.choice(["fp32", "fp32", "ue8m0"])
            case = _moe(_log_uniform(rng, 1, 4096), e, h, i, topk, checkpoint)
        else:
            max_m = rng.choice([64, 128, 256])
            case = _masked(rng.choice([16, 32]), max_m, _log_uniform(rng, 1, max_m // 2), rng.choice([4096, 7168]),
                           rng.choice([1536, 2048]))
        if work(case)["flops"] <= LARGEST_FLOPS:
            return case


def _activations(g, rows, cols, dtype):
    x = torch.randn(rows, cols, generator=g, device="cuda")
    outlier = torch.rand(rows, cols, generator=g, device="cuda") < 0.01
    return torch.where(outlier, x * 50, x).to(dtype)


def _expert_weights(g, experts, n, k, checkpoint):
    """Codes and block scales of ~N(0, 0.02) weights, drawn directly in quantised form (a block's largest code is near
    448): fp32 scales, or packed powers of two."""
    w = torch.empty(experts, n, k, dtype=torch.float8_e4m3fn, device="cuda")
    for e0 in range(0, experts, 8):
        part = w[e0:e0 + 8]
        part.copy_(torch.randn(part.shape, generator=g, device="cuda").mul_(110).clamp_(-448, 448))
    shape = (experts, -(-n // 128), -(-k // 128))
    if checkpoint == "fp32":
        return w, (torch.rand(shape, generator=g, device="cuda") * 0.2 + 0.9) * (0.02 / 110)
    s = torch.exp2(torch.randint(-13, -11, shape, generator=g, device="cuda").float())
    return w, pack_ue8m0_scales(s.view(-1, shape[2])).view(experts, shape[1], -1)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return {"linear": _prepare_linear, "quant": _prepare_quant, "moe": _prepare_moe,
            "masked": _prepare_masked}[case["op"]](case, g)


def _prepare_linear(case, g):
    m, n, k, dtype = case["m"], case["n"], case["k"], DTYPES[case["dtype"]]
    layer = torch.nn.Module()
    method = Fp8LinearMethod(Fp8Config())
    method.create_weights(layer, k, [n], k, n, dtype, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda").mul_(0.02)
    codes, scales = block_quant_weight_fp8(w) if case["checkpoint"] == "fp32" else per_block_cast_to_fp8(w)
    layer.weight.data.copy_(codes)
    layer.weight_scale_inv.data.copy_(scales)
    method.process_weights_after_loading(layer)
    bias = torch.randn(n, generator=g, device="cuda").to(dtype) if case["bias"] else None
    return {"op": "linear", "method": method, "layer": layer, "x": _activations(g, m, k, dtype), "bias": bias}


def _prepare_quant(case, g):
    cols = case["k"] * (2 if case["silu"] else 1)
    x = torch.randn(case["m"], cols, generator=g, device="cuda")
    if not case["silu"]:
        x *= torch.pow(10.0, torch.rand(case["m"], 1, generator=g, device="cuda") * 4 - 2)
    layout = case["layout"]
    options = {"column_major_scales": layout != "row", "scale_tma_aligned": layout in ("col_tma", "ue8m0"),
               "scale_ue8m0": layout == "ue8m0", "fuse_silu_and_mul": case["silu"]}
    return {"op": "quant", "x": x.to(DTYPES[case["dtype"]]), "options": options}


def _prepare_moe(case, g):
    m, e, h, i = case["m"], case["experts"], case["hidden"], case["inter"]
    w1, s1 = _expert_weights(g, e, 2 * i, h, case["checkpoint"])
    w2, s2 = _expert_weights(g, e, h, i, case["checkpoint"])
    return {"op": "moe", "checkpoint": case["checkpoint"], "topk": case["topk"],
            "x": torch.randn(m, h, generator=g, device="cuda").to(torch.bfloat16),
            "logits": torch.randn(m, e, generator=g, device="cuda"), "w1": w1, "s1": s1, "w2": w2, "s2": s2,
            "gate_bias": torch.randn(e, generator=g, device="cuda") * 0.1, "groups": 8 if e >= 64 else 1,
            "config": MoeRunnerConfig(num_experts=e, top_k=case["topk"])}


def _prepare_masked(case, g):
    e, max_m, h, i = case["experts"], case["max_m"], case["hidden"], case["inter"]
    slots = torch.randint(0, e, (e * case["expected_m"],), generator=g, device="cuda")
    masked_m = torch.bincount(slots, minlength=e).clamp(max=max_m).to(torch.int32)
    x = torch.randn(e, max_m, h, generator=g, device="cuda").to(torch.bfloat16)
    w1, s1 = _expert_weights(g, e, 2 * i, h, "fp32")
    w2, s2 = _expert_weights(g, e, h, i, "fp32")
    return {"op": "masked", "a": sglang_per_token_group_quant_fp8(x, 128), "w1": (w1, s1), "w2": (w2, s2),
            "masked_m": masked_m, "expected_m": case["expected_m"],
            "gate_up": torch.zeros(e, max_m, 2 * i, dtype=torch.bfloat16, device="cuda"),
            "out": torch.zeros(e, max_m, h, dtype=torch.bfloat16, device="cuda")}


def run(state):
    op = state["op"]
    if op == "linear":
        return state["method"].apply(state["layer"], state["x"], state["bias"])
    if op == "quant":
        return sglang_per_token_group_quant_fp8(state["x"], 128, **state["options"])
    if op == "masked":
        m, expected = state["masked_m"], state["expected_m"]
        grouped_gemm_nt_f8f8bf16_masked(state["a"], state["w1"], state["gate_up"], m, expected)
        down = sglang_per_token_group_quant_fp8(state["gate_up"], 128, fuse_silu_and_mul=True, masked_m=m)
        grouped_gemm_nt_f8f8bf16_masked(down, state["w2"], state["out"], m, expected)
        return state["out"]
    x, logits, topk = state["x"], state["logits"], state["topk"]
    if state["checkpoint"] == "fp32":
        weights, ids = fused_topk(x, logits, topk, True)
        out = fused_experts(x, state["w1"], state["w2"], StandardTopKOutput(weights, ids, logits), state["config"],
                            use_fp8_w8a8=True, w1_scale=state["s1"], w2_scale=state["s2"], block_shape=[128, 128])
    else:
        weights, ids = biased_grouped_topk(x, logits, state["gate_bias"], topk, True, state["groups"],
                                           max(1, state["groups"] // 2), routed_scaling_factor=2.5)
        out = fused_experts_block_fp8_ue8m0(x, state["w1"], state["w2"], state["s1"], state["s2"], weights, ids)
    return {"out": out, "weights": weights, "ids": ids}


def work(case):
    if case["op"] == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        scales = -(-n // 128) * -(-k // 128) * (4 if case["checkpoint"] == "fp32" else 1)
        return {"bytes": 2 * m * k + n * k + scales + 2 * m * n + (2 * n if case["bias"] else 0), "flops": 2 * m * n * k}
    if case["op"] == "quant":
        m, k = case["m"], case["k"]
        scale = 1 if case["layout"] == "ue8m0" else 4
        return {"bytes": (4 if case["silu"] else 2) * m * k + m * k + m * k // 128 * scale, "flops": 0}
    e, h, i = case["experts"], case["hidden"], case["inter"]
    if case["op"] == "masked":
        rows = e * case["expected_m"]
        used = e * (1 - (1 - 1 / e) ** rows)
        return {"bytes": used * 3 * h * i + rows * (h + h // 32 + 2 * h), "flops": 6 * rows * h * i}
    m, topk = case["m"], case["topk"]
    used = e * (1 - (1 - topk / e) ** m)
    return {"bytes": used * 3 * h * i + 4 * m * h + 4 * m * e + 8 * m * topk, "flops": 6 * m * topk * h * i}


def tolerance(case):
    if case["op"] == "quant":
        # codes and scales are whole results; behind the SiLU one rounding of the activation can move a code by one
        return {"rel": 2e-3, "max": 0.15, "differ": 1e-3} if case["silu"] else "exact"
    if case["op"] == "linear":
        return {"rel": 1e-2, "max": 2e-2}  # 16-bit results of 32-bit sums
    return {"rel": 1e-2, "max": 5e-2, "differ": 1e-3}  # the activations are quantised once more between the two GEMMs
