"""The calls that the framework's speed is judged by: what an engine does with one fused-MoE layer.

A case is one call of a public op of ``aklr_b200.ops`` on one GPU, or the replay of a CUDA graph that holds that one
call, as a serving engine runs its decode batches.  The widths are those of ``aklr_b200.workloads.CONFIGS``, of
``bench.py``'s recorded workloads and of their tensor-parallel slices; token counts run from one (decode) to a long
prefill.  Every input is made from the seed: activations N(0, 1) in bf16, expert weights N(0, 0.02) in the checkpoint's
format, router weights that give logits of about unit variance.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from aklr_b200 import ops
from aklr_b200 import workloads as wl

BF16 = torch.bfloat16


def listed():
    return [
        # one user's decode step of the widest layer: 9 experts' weights and five launches, replayed from the engine's graph
        dict(name="deepseek_fp8_t1_graph", op="deepseek_v2_fp8_moe", tokens=1, hidden=7168, inter=2048, routed=256, topk=8, graph=True),
        # a decode batch of the same layer called eagerly: most of the 11 GB of weights are read for a few rows each
        dict(name="deepseek_fp8_t64", op="deepseek_v2_fp8_moe", tokens=64, hidden=7168, inter=2048, routed=256, topk=8, graph=False),
        # a prefill chunk of it, the benchmark's own size: 128 rows for each routed expert, 4096 for the shared one
        dict(name="deepseek_fp8_t4096", op="deepseek_v2_fp8_moe", tokens=4096, hidden=7168, inter=2048, routed=256, topk=8, graph=False),
        # the longest prefill of an eighth of it (tensor parallel over 8): long rows, short inner width
        dict(name="deepseek_fp8_tp8_t16384", op="deepseek_v2_fp8_moe", tokens=16384, hidden=7168, inter=256, routed=256, topk=8, graph=False),
        # few large experts, softmax routing to two of eight: a mid-sized prefill
        dict(name="mixtral_fp8_t1024", op="qwen3_moe_fp8_moe", tokens=1024, hidden=4096, inter=14336, routed=8, topk=2, graph=False),
        # many small experts, popularity skewed, an odd count of tokens between decode and prefill
        dict(name="qwen3_fp8_t333", op="qwen3_moe_fp8_moe", tokens=333, hidden=2048, inter=768, routed=128, topk=8, graph=False, zipf=1.1),
        # float32 router, a tensor-parallel slice, a ragged prefill
        dict(name="minimax_fp8_t2000", op="minimax_m2_fp8_moe", tokens=2000, hidden=3072, inter=384, routed=256, topk=8, graph=False),
        # the smallest experts, gated shared expert, a small odd decode batch: launches and host work
        dict(name="qwen2_fp8_t17", op="qwen2_moe_fp8_router_experts", tokens=17, hidden=2048, inter=128, routed=512, topk=10, graph=False),
        # experts-only op on MXFP4 weights at its default (MXFP4 activations), a decode batch in a graph
        dict(name="fused_mxfp4_a4_t64_graph", op="fused_moe", tokens=64, hidden=6144, inter=256, routed=257, topk=9, graph=True, act_quant=4),
        # MXFP4 weights with MXFP8 activations at full width, the benchmark's size: the most arithmetic in one call
        dict(name="fused_mxfp4_a8_t8192", op="fused_moe", tokens=8192, hidden=7168, inter=2048, routed=257, topk=9, graph=False, act_quant=8),
        # MXFP4 weights with activations left in bf16, router included, an odd prefill
        dict(name="deepseek_mxfp4_t1001", op="deepseek_v2_mxfp4_moe", tokens=1001, hidden=6144, inter=256, routed=256, topk=8, graph=False),
        # the stand-alone activation quantiser that feeds an engine's dense FP8 GEMMs
        dict(name="quant_fp8_r2048", op="per_group_quant_fp8", tokens=2048, hidden=7168, graph=False),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    family = rng.choice(["deepseek", "deepseek", "mixtral", "qwen3", "minimax", "qwen2", "fused", "fused", "deepseek_mx", "quant"])
    if family == "quant":
        return dict(op=rng.choice(["per_group_quant_fp8", "per_group_quant_mxfp8"]), tokens=_log_int(rng, 16, 16384),
                    hidden=128 * rng.randint(8, 56), graph=False)
    if family == "deepseek":
        case = dict(op="deepseek_v2_fp8_moe", hidden=7168, inter=rng.choice([256, 512, 1024, 2048]), routed=256, topk=8)
    elif family == "mixtral":
        case = dict(op="qwen3_moe_fp8_moe", hidden=4096, inter=rng.choice([1792, 3584, 7168, 14336]), routed=8, topk=2)
    elif family == "qwen3":
        case = dict(op="qwen3_moe_fp8_moe", hidden=2048, inter=rng.choice([384, 768]), routed=128, topk=8, zipf=1.1)
    elif family == "minimax":
        case = dict(op="minimax_m2_fp8_moe", hidden=3072, inter=rng.choice([384, 768, 1536]), routed=256, topk=8)
    elif family == "qwen2":
        case = dict(op="qwen2_moe_fp8_router_experts", hidden=2048, inter=rng.choice([128, 256, 512]), routed=512, topk=10)
    elif family == "fused":
        case = dict(op="fused_moe", hidden=rng.choice([6144, 7168]), inter=rng.choice([256, 512, 1024, 2048]), routed=257, topk=9,
                    act_quant=rng.choice([4, 8]))
    else:
        case = dict(op="deepseek_v2_mxfp4_moe", hidden=6144, inter=rng.choice([256, 512]), routed=256, topk=8)
    most = 16384
    budget = 1.6e12 if case["op"] == "deepseek_v2_mxfp4_moe" else 3.2e12  # operations of the largest listed call of this kind
    while 6 * most * _routes(case) * case["hidden"] * case["inter"] > budget:
        most //= 2
    case["tokens"] = _log_int(rng, 1, most)
    case["graph"] = case["tokens"] <= 256 and rng.random() < 0.5
    return case


def _routes(case):
    """Experts a token goes to, the shared one included."""
    return case["topk"] + (case["op"].startswith(("deepseek", "qwen2")))


def _experts(case):
    return case["routed"] + (case["op"].startswith(("deepseek", "qwen2")))


def _is_mx(case):
    return case["op"] in ("fused_moe", "deepseek_v2_mxfp4_moe")


def _router(case, seed, device, dtype):
    """A router whose logits on N(0, 1) activations have unit variance."""
    return wl.normal(seed, "router", (case["routed"], case["hidden"]), case["hidden"] ** -0.5, device, dtype)


def _skewed(case, x, router, seed):
    """Activations with a component along a direction that the router answers with -s ln(rank): Zipf popularity."""
    ranks = 1.0 + torch.randperm(case["routed"], generator=torch.Generator().manual_seed(seed % (1 << 62))).to(torch.float32)
    common = wl.normal(seed, "common", (case["hidden"],), 1.0, x.device)
    common /= common.norm()
    x = (x.float() + 4.0 * common).to(BF16)
    popularity = (-case["zipf"] * ranks.log()).to(x.device)
    return x, (router.float() + torch.outer((popularity - popularity.mean()) / 4.0, common)).to(BF16)


def _arguments(case, seed, device):
    tokens, hidden = case["tokens"], case["hidden"]
    x = wl.normal(seed, "hidden", (tokens, hidden), 1.0, device, BF16)
    if case["op"].startswith("per_group_quant"):
        return dict(x=x)
    cfg = wl.MoEConfig(case["op"], hidden=hidden, inter=case["inter"], n_routed=_experts(case), topk=case["topk"])
    w1, s1, w2, s2 = (wl.mx_expert_weights if _is_mx(case) else wl.expert_weights)(cfg, seed, device)
    call = dict(hidden_states=x, w1=w1, w1_scale=s1, w2=w2, w2_scale=s2)
    if case["op"] == "fused_moe":
        scores = wl.normal(seed, "scores", (tokens, case["routed"]), 1.0, device)
        top = scores.topk(case["topk"], dim=-1)
        call.update(topk_ids=top.indices.to(torch.int32), topk_weights=top.values.softmax(-1), activation="silu",
                    quant_type="per_1x32", act_quant=case["act_quant"])
        return call
    call["topk"] = case["topk"]
    if case["op"] == "minimax_m2_fp8_moe":
        call["router_weight"] = _router(case, seed, device, torch.float32)
        call["correction_bias"] = wl.normal(seed, "bias", (case["routed"],), 0.01, device)
        return call
    call["router_weight"] = _router(case, seed, device, BF16)
    if case["op"].startswith("deepseek"):
        fp8 = case["op"] == "deepseek_v2_fp8_moe"
        call["correction_bias"] = wl.normal(seed, "bias", (case["routed"],), 0.01, device, BF16 if fp8 else torch.float32)
        call.update(num_expert_group=8 if fp8 else 1, topk_group=4 if fp8 else 1, renormalize=True, scoring_func="sigmoid",
                    routed_scaling_factor=2.5)
    elif case["op"].startswith("qwen2"):
        call["shared_gate_weight"] = wl.normal(seed, "shared_gate", (1, hidden), hidden**-0.5, device, BF16)
    if case.get("zipf"):
        call["hidden_states"], call["router_weight"] = _skewed(case, x, call["router_weight"], seed)
    return call


def _call(state):
    out = state["op"](**state["call"])
    if isinstance(out, ops.FallbackReason):
        raise RuntimeError(f"{state['op'].__name__} was not served: {out}")
    return out


def prepare(case, seed):
    ops.init()
    state = dict(op=getattr(ops, case["op"]), call=_arguments(case, seed, torch.device("cuda", torch.cuda.current_device())), graph=None)
    if case["graph"]:
        _call(state)  # an engine calls each batch size once before it captures it
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = _call(state)
    return state


def run(state):
    if state["graph"] is not None:
        state["graph"].replay()
        return state["out"]
    return _call(state)


@functools.lru_cache(maxsize=None)
def _experts_hit(routed, topk, tokens, zipf):
    """Distinct routed experts a batch reaches: expected under even popularity, one simulated batch under a skewed one."""
    if not zipf:
        return routed * (1.0 - (1.0 - topk / routed) ** tokens)
    rng = np.random.default_rng(1)
    logits = rng.standard_normal((min(tokens, 4096), routed)) - zipf * np.log(np.arange(1, routed + 1))
    return float(np.unique(np.argpartition(-logits, topk - 1, axis=1)[:, :topk]).size)


def work(case):
    tokens, hidden = case["tokens"], case["hidden"]
    if case["op"].startswith("per_group_quant"):
        scale = hidden // 128 * 4 if case["op"].endswith("_fp8") else hidden // 32
        return {"bytes": tokens * (3 * hidden + scale), "flops": 0}
    inter, shared = case["inter"], _experts(case) - case["routed"]
    weights = 3 * hidden * inter
    expert = weights / 2 + weights / 32 if _is_mx(case) else weights + weights / 128**2 * 4
    hit = _experts_hit(case["routed"], case["topk"], tokens, case.get("zipf", 0.0)) + shared
    router = 0 if case["op"] == "fused_moe" else case["routed"] * hidden * (4 if case["op"].startswith("minimax") else 2)
    routing = tokens * case["topk"] * 8 if case["op"] == "fused_moe" else 0
    return {
        "bytes": hit * expert + router + routing + tokens * hidden * 4,
        "flops": 2 * tokens * _routes(case) * weights + (2 * tokens * hidden * case["routed"] if router else 0),
    }


def tolerance(case):
    if case["op"].startswith("per_group_quant"):
        return "exact"
    # Against the same layer summed in 64 bits on the same routing: 0.0023 .. 0.0036 relative, at most 0.06 of a value (bf16
    # route rows and output, gated products that round to a neighbouring code); four times that.
    return {"rel": 0.012, "max": 0.25}
