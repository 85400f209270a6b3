"""The calls a serving stack makes of the fused Mixture-of-Experts layer, as cases for timing.

Layers, token counts and value distributions are those of the repository's own configurations
(``flaggems_sglang_b200.testing.CONFIGS`` and the benchmark's sweeps): weights ``randn * 0.02``, unit
normal activations, top-k of a softmax over the router's logits, with the zipf-skewed router for the
256-expert layer.  A case is

    layer    name in CONFIGS
    weights  "bf16" | "fp16" | "fp8" (e4m3, 128x128 block scales) | "int4" (AWQ w4a16, groups of 128)
    tokens   rows of the batch
    entry    "hook"     the serving stack's plug-in hook, from top-k ids and weights
             "experts"  the layer-layout operator, from top-k ids and weights
             "logits"   router and experts in one call, from the gating logits
             "op"       the reference's operator with its routing conversion in front
             "op_bias"  the same with per-expert biases and the clamped swiglu
    graph    the call is captured in a CUDA graph once and a pass replays it, as decode steps are served
"""
import math
import sys
from pathlib import Path
from types import SimpleNamespace

import torch

_ROOT = Path(__file__).resolve().parent.parent
for _p in (Path.cwd() / "flaggems-sglang_b200", _ROOT / "flaggems-sglang_b200"):
    if _p.is_dir():                       # the tree that is the working folder comes first
        sys.path.insert(0, str(_p))
        break

import flaggems_sglang_b200 as F  # noqa: E402
from flaggems_sglang_b200.quant import quantize_awq, quantize_fp8_block, repack_awq_for_kernel  # noqa: E402
from flaggems_sglang_b200.testing import CONFIGS, route, zipf_bias  # noqa: E402

_TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp8": torch.bfloat16, "int4": torch.float16}
_WEIGHT_BYTES = {"bf16": 2.0, "fp16": 2.0, "fp8": 1.0, "int4": 0.5}


def _case(name, layer, weights, tokens, entry, graph=False):
    return {"name": name, "layer": layer, "weights": weights, "tokens": tokens, "entry": entry, "graph": graph}


def listed():
    return [
        # one user's decode step through the plug-in hook: eight small experts, launches and host time count
        _case("many-experts one token", "qwen3-30b-a3b", "bf16", 1, "hook"),
        # a small decode batch, router included, replayed from a CUDA graph
        _case("many-experts decode graph", "qwen3-30b-a3b", "bf16", 32, "logits", graph=True),
        # a full decode batch of odd size: nearly every expert holds a few tokens
        _case("many-experts decode", "qwen3-30b-a3b", "bf16", 201, "hook"),
        # decode with few large experts: all weights stream once
        _case("large-experts decode", "mixtral", "bf16", 16, "experts"),
        # a short prompt or a chunk of prefill: ragged token blocks, memory and tensor cores both loaded
        _case("large-experts short prefill", "mixtral", "bf16", 1000, "experts"),
        # the benchmark's own workload
        _case("large-experts prefill", "mixtral", "bf16", 4096, "hook"),
        # the reference's benchmark shapes through its own operator, with the routing conversion in front
        _case("operator decode", "reference-bench", "bf16", 17, "op"),
        _case("operator prefill", "reference-bench", "bf16", 2048, "op"),
        # block-quantised FP8 layer with 256 unevenly hit experts
        _case("fp8 decode", "deepseek-v3", "fp8", 64, "experts"),
        _case("fp8 prefill", "deepseek-v3", "fp8", 4096, "experts"),
        # int4 AWQ layer
        _case("int4 decode", "mixtral", "int4", 32, "experts"),
        _case("int4 prefill", "mixtral", "int4", 2048, "experts"),
    ]


def draw(rng):
    weights, layer = rng.choice([("bf16", "qwen3-30b-a3b"), ("bf16", "mixtral"), ("bf16", "reference-bench"),
                                 ("fp16", "qwen3-30b-a3b"), ("fp16", "mixtral"), ("fp8", "deepseek-v3"),
                                 ("fp8", "deepseek-v3"), ("int4", "mixtral"), ("int4", "mixtral")])
    most = 2048 if weights == "int4" else 4096
    tokens = max(1, min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1.0))))))
    if layer == "reference-bench":
        entry = rng.choice(["op", "op", "op_bias"])
    elif weights in ("bf16", "fp16"):
        entry = rng.choice(["hook", "experts", "logits"])
    else:
        entry = rng.choice(["experts", "logits"])
    graph = tokens <= 256 and rng.random() < 0.3
    return {"layer": layer, "weights": weights, "tokens": tokens, "entry": entry, "graph": graph}


def _weights(case, gen):
    """The layer's weights as the case's entry point takes them."""
    h, i, e, _ = CONFIGS[case["layer"]]
    kind, dtype = case["weights"], _TYPES[case["weights"]]

    def rand(rows, cols):
        return torch.randn(rows, cols, generator=gen, device="cuda", dtype=dtype).mul_(0.02)

    if kind == "fp8":
        w13 = torch.empty(e, 2 * i, h, dtype=torch.float8_e4m3fn, device="cuda")
        w2 = torch.empty(e, h, i, dtype=torch.float8_e4m3fn, device="cuda")
        s13 = torch.empty(e, -(-2 * i // 128), -(-h // 128), device="cuda")
        s2 = torch.empty(e, -(-h // 128), -(-i // 128), device="cuda")
        for x in range(e):
            q, s = quantize_fp8_block(rand(2 * i, h)[None])
            w13[x], s13[x] = q[0], s[0]
            q, s = quantize_fp8_block(rand(h, i)[None])
            w2[x], s2[x] = q[0], s[0]
        return {"w13": w13, "w2": w2, "kw": dict(use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2)}
    if kind == "int4":
        got = [[], [], [], []]
        for x in range(e):
            for at, (k, n) in ((0, (h, 2 * i)), (2, (i, h))):
                p, z = repack_awq_for_kernel(*quantize_awq(rand(k, n)[None]))
                got[at].append(p)
                got[at + 1].append(z)
        w13, z13, w2, z2 = (torch.cat(g) for g in got)
        return {"w13": w13, "w2": w2, "kw": dict(use_int4_w4a16=True, w13_sz=z13, w2_sz=z2)}
    op = case["entry"] in ("op", "op_bias")             # the reference's operator: [E, H, 2I] and [E, I, H]
    w13 = torch.empty((e, h, 2 * i) if op else (e, 2 * i, h), dtype=dtype, device="cuda")
    w2 = torch.empty((e, i, h) if op else (e, h, i), dtype=dtype, device="cuda")
    for x in range(e):
        w13[x] = rand(*w13.shape[1:])
        w2[x] = rand(*w2.shape[1:])
    got = {"w13": w13, "w2": w2, "kw": {}}
    if case["entry"] == "op_bias":
        for name, n in (("b13", 2 * i), ("b2", h)):
            got[name] = torch.randn(e, n, generator=gen, device="cuda").mul_(0.1)
    return got


def _hold(module, **params):
    for name, t in params.items():
        setattr(module, name, torch.nn.Parameter(t, requires_grad=False))
    return module


def prepare(case, seed):
    h, i, e, k = CONFIGS[case["layer"]]
    m = case["tokens"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = _weights(case, gen)
    s["entry"], s["topk"], s["experts"] = case["entry"], k, e
    s["x"] = torch.randn(m, h, generator=gen, device="cuda", dtype=_TYPES[case["weights"]])
    s["logits"] = torch.randn(m, e, generator=gen, device="cuda")
    if case["layer"] == "deepseek-v3":
        s["logits"] += zipf_bias(e, 1.1, seed=0).cuda()
    s["tw"], s["ids"] = route(s["logits"], k)
    if case["entry"] == "hook":
        s["layer"] = _hold(torch.nn.Module(), w13_weight=s["w13"], w2_weight=s["w2"])
        config = SimpleNamespace(activation="silu", apply_router_weight_on_input=False, no_combine=False,
                                 routed_scaling_factor=None)
        s["obj"] = SimpleNamespace(runner=SimpleNamespace(config=config))
        s["dispatch"] = SimpleNamespace(hidden_states=s["x"],
                                        topk_output=SimpleNamespace(topk_weights=s["tw"], topk_ids=s["ids"]))
    if case["graph"]:
        _call(s)                                        # loads the library and sizes its scratch
        torch.cuda.synchronize()
        s["replay"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["replay"]):
            s["out"] = _call(s)
    return s


def _call(s):
    entry = s["entry"]
    if entry == "hook":
        return F.fused_moe_flagos(s["obj"], s["layer"], s["dispatch"]).hidden_states
    if entry == "experts":
        return F.fused_experts(s["x"], s["w13"], s["w2"], s["tw"], s["ids"], **s["kw"])
    if entry == "logits":
        return F.fused_moe(s["x"], s["w13"], s["w2"], s["logits"], s["topk"], **s["kw"])
    routing = F.topk_to_routing(s["tw"], s["ids"], s["experts"])
    if entry == "op":
        return F.triton_kernel_fused_experts(s["x"], s["w13"], s["w2"], *routing)
    return F.triton_kernel_fused_experts_with_bias(s["x"], s["w13"], None, s["b13"], s["w2"], None, s["b2"], *routing,
                                                   gemm1_alpha=1.702, gemm1_clamp_limit=7.0)


def run(state):
    if "replay" in state:
        state["replay"].replay()
        return state["out"]
    return _call(state)


def _experts_hit(case):
    """Experts that hold at least one token, on average over the router's draws."""
    _, _, e, k = CONFIGS[case["layer"]]
    m = case["tokens"]
    if case["layer"] != "deepseek-v3":
        return e * (1.0 - (1.0 - k / e) ** m)
    gen = torch.Generator().manual_seed(1)
    logits = torch.randn(m, e, generator=gen) + zipf_bias(e, 1.1, seed=0)
    return float(torch.topk(logits, k, dim=-1).indices.unique().numel())


def work(case):
    h, i, _, k = CONFIGS[case["layer"]]
    m = case["tokens"]
    expert = 3.0 * h * i * _WEIGHT_BYTES[case["weights"]]
    if case["weights"] == "fp8":
        expert += 3.0 * h * i / (128 * 128) * 4         # an fp32 scale per 128x128 block
    elif case["weights"] == "int4":
        expert += 3.0 * h * i / 128 * 2.5               # fp16 scale and 4-bit zero per row and group
    return {"bytes": _experts_hit(case) * expert + m * h * 4.0, "flops": 6.0 * m * k * h * i}


def tolerance(case):
    # results and intermediates are 16-bit; sums run in fp32 in whatever order
    return {"rel": 2e-3 if case["weights"] in ("fp16", "int4") else 1e-2}
