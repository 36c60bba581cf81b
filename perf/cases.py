"""The work that users of this package have it do, as cases that can be timed: one MoE layer call each.

A layer is one of the shapes that `workloads.py` and the tests hold (hidden size H, intermediate size I, E experts,
top-k, weight format), a token count T from a single decoded token to a prefill of thousands, and the entry point that
a program of that kind calls:

  moe     fused_moe(hidden, w1, w2, router logits): the serving-side layer, router included
  triple  triton_kernel_fused_experts(hidden, w1 [E,H,2I], w2 [E,I,H], routing triple): the reference's operator, with
          weights in its own layout
  hook    fused_moe_flagos(obj, layer, dispatch_output): the serving hook, on already routed tokens

`tp` divides I, as a tensor-parallel rank holds it.  `skew` draws the router logits with a Zipf(1.2) bias, so that some
experts are hot and some get next to nothing.
"""
import math
from types import SimpleNamespace

import torch

import flaggems_sglang_b200 as fg

# H, I, E, top-k, weight format, router; most tokens a call has
LAYERS = {
    "mixtral": dict(H=4096, I=14336, E=8, k=2, fmt="bf16", most=4096),
    "qwen3": dict(H=2048, I=768, E=128, k=8, fmt="bf16", most=8192),
    "dsv3": dict(H=7168, I=2048, E=256, k=8, fmt="fp8_block", most=4096, groups=(8, 4), factor=2.5),
    "dsv3_channel": dict(H=7168, I=2048, E=256, k=8, fmt="fp8_channel", most=4096, groups=(8, 4), factor=2.5),
    "refbench": dict(H=1280, I=3072, E=64, k=8, fmt="bf16", most=4096),
    "gpt_oss": dict(H=2880, I=2880, E=32, k=4, fmt="bf16", most=4096, bias=True),
}


def _case(name, layer, T, entry="moe", tp=1, skew=False):
    return dict(name=name, layer=layer, T=T, entry=entry, tp=tp, skew=skew)


def listed():
    return [
        # one user's decode step: 75 MB of weights, launches and latency are a large share
        _case("qwen3 decode 1", "qwen3", 1),
        # the same for a large fp8 layer behind the grouped router
        _case("dsv3 decode 1", "dsv3", 1),
        # an odd, small decode batch on a layer with few, wide experts
        _case("mixtral decode 19", "mixtral", 19),
        # the reference's own test and benchmark list, through its operator: many small experts
        _case("refbench op 17", "refbench", 17, entry="triple"),
        # a large fp8 decode batch: every expert has a few rows
        _case("dsv3 decode 128", "dsv3", 128),
        # a chunk of mixed prefill and decode on one tensor-parallel rank, through the serving hook
        _case("mixtral hook 333 tp2", "mixtral", 333, entry="hook", tp=2),
        # biases and the clamped swiglu, sizes that no tile divides, through the serving hook
        _case("gpt_oss hook 700", "gpt_oss", 700, entry="hook"),
        # the reference's largest test shape, through its operator
        _case("refbench op 1024", "refbench", 1024, entry="triple"),
        # per-channel fp8 prefill chunk
        _case("dsv3_channel prefill 2048", "dsv3_channel", 2048),
        # long prefill, skewed routing, ragged token count
        _case("qwen3 prefill 7777 skew", "qwen3", 7777, skew=True),
        # the benchmark's own point
        _case("mixtral prefill 4096", "mixtral", 4096),
        # fp8 prefill with 128x128 block scales
        _case("dsv3 prefill 4096", "dsv3", 4096),
    ]


def draw(rng):
    # every layer, entry point and token count of the list's ranges
    layer = rng.choice(sorted(LAYERS))
    L = LAYERS[layer]
    tp = rng.choice([1, 1, 2, 4])
    while (L["I"] // tp) % (128 if L["fmt"] == "fp8_block" else 32) or L["I"] % tp:
        tp //= 2
    if L.get("bias"):
        entry = "hook"
    elif L["fmt"] != "bf16":
        entry = "moe"
    else:
        entry = rng.choice(["moe", "moe", "triple", "hook"])
    T = int(round(math.exp(rng.uniform(0.0, math.log(L["most"])))))
    return dict(layer=layer, T=max(1, min(T, L["most"])), entry=entry, tp=tp, skew=rng.random() < 0.25)


def _weights(L, I, gen, dev, n_major):
    """N(0,1)/sqrt(fan-in) weights, an expert at a time so that little is held in fp32."""
    H, E, fmt = L["H"], L["E"], L["fmt"]
    wdt = torch.bfloat16 if fmt == "bf16" else torch.float8_e4m3fn
    s1, s2 = ((2 * I, H), (H, I)) if not n_major else ((H, 2 * I), (I, H))
    w1 = torch.empty(E, *s1, dtype=wdt, device=dev)
    w2 = torch.empty(E, *s2, dtype=wdt, device=dev)
    scales = []
    for e in range(E):
        a = torch.randn(*s1, generator=gen, device=dev, dtype=torch.float32).mul_(1.0 / math.sqrt(H))
        b = torch.randn(*s2, generator=gen, device=dev, dtype=torch.float32).mul_(1.0 / math.sqrt(I))
        if fmt == "bf16":
            w1[e], w2[e] = a, b
        else:
            quant = fg.quant_weight_block128 if fmt == "fp8_block" else fg.quant_weight_per_channel
            w1[e], sa = quant(a)
            w2[e], sb = quant(b)
            scales.append((sa, sb))
    if not scales:
        return w1, w2, None, None
    return w1, w2, torch.stack([s[0] for s in scales]), torch.stack([s[1] for s in scales])


def prepare(case, seed):
    dev = torch.device("cuda")
    L = LAYERS[case["layer"]]
    H, I, E, k, T = L["H"], L["I"] // case["tp"], L["E"], L["k"], case["T"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    w1, w2, s1, s2 = _weights(L, I, gen, dev, case["entry"] == "triple")
    hidden = torch.randn(T, H, generator=gen, device=dev, dtype=torch.float32).to(torch.bfloat16)
    logits = torch.randn(T, E, generator=gen, device=dev, dtype=torch.float32)
    if case["skew"]:
        rank = torch.randperm(E, generator=gen, device=dev).float() + 1.0
        logits += torch.log(rank.pow(-1.2) / rank.pow(-1.2).sum())
    state = dict(entry=case["entry"], hidden=hidden, w1=w1, w2=w2, logits=logits, k=k)
    if case["entry"] == "moe":
        kw = {}
        if L["fmt"] == "fp8_block":
            kw.update(use_fp8_w8a8=True, block_shape=[128, 128], w1_scale=s1, w2_scale=s2)
        elif L["fmt"] == "fp8_channel":
            kw.update(use_fp8_w8a8=True, per_channel_quant=True, w1_scale=s1, w2_scale=s2)
        if "groups" in L:
            bias = torch.randn(E, generator=gen, device=dev, dtype=torch.float32) * 0.1
            kw.update(use_grouped_topk=True, num_expert_group=L["groups"][0], topk_group=L["groups"][1],
                      correction_bias=bias, routed_scaling_factor=L["factor"])
        state["kw"] = kw
        return state
    weights, ids = fg.fused_topk(hidden, logits, k, True)
    if case["entry"] == "triple":
        state["routing"] = fg.standard_topk_to_routing(weights, ids, E)
        return state
    layer = SimpleNamespace(w13_weight=w1, w2_weight=w2)
    if L.get("bias"):
        layer.w13_weight_bias = torch.randn(E, 2 * I, generator=gen, device=dev, dtype=torch.float32) * 0.1
        layer.w2_weight_bias = torch.randn(E, H, generator=gen, device=dev, dtype=torch.float32) * 0.1
    config = SimpleNamespace(num_experts=E, activation="silu", apply_router_weight_on_input=False, no_combine=False,
                             routed_scaling_factor=None, gemm1_alpha=1.702, gemm1_clamp_limit=7.0)
    state["obj"] = SimpleNamespace(runner=SimpleNamespace(config=config))
    state["layer"] = layer
    state["dispatch"] = SimpleNamespace(hidden_states=hidden,
                                        topk_output=SimpleNamespace(topk_weights=weights, topk_ids=ids))
    return state


def run(state):
    if state["entry"] == "moe":
        return fg.fused_moe(state["hidden"], state["w1"], state["w2"], state["logits"], state["k"], True, **state["kw"])
    if state["entry"] == "triple":
        return fg.triton_kernel_fused_experts(state["hidden"], state["w1"], state["w2"], *state["routing"])
    return fg.fused_moe_flagos(state["obj"], state["layer"], state["dispatch"]).hidden_states


def _active_experts(case):
    """Experts that get rows in one sampled routing of such a call (the sample holds up to 2048 tokens: past that every
    expert that gets any has got some)."""
    L = LAYERS[case["layer"]]
    E, k, T = L["E"], L["k"], min(case["T"], 2048)
    gen = torch.Generator().manual_seed(1)
    score = torch.randn(T, E, generator=gen)
    if case["skew"]:
        rank = torch.randperm(E, generator=gen).float() + 1.0
        score += torch.log(rank.pow(-1.2) / rank.pow(-1.2).sum())
    if "groups" in L:
        score = torch.sigmoid(score) + torch.randn(E, generator=gen) * 0.1
        groups, kept = L["groups"]
        best = score.view(T, groups, -1).topk(2, dim=2).values.sum(2).topk(kept, dim=1).indices
        keep = torch.zeros(T, groups).scatter_(1, best, 1.0).repeat_interleave(E // groups, dim=1)
        score = score.masked_fill(keep == 0.0, -math.inf)
    return int(score.topk(k, dim=1).indices.unique().numel())


def work(case):
    """Hidden states, logits (or routing) and the weights of the experts that get rows, read once; the output written
    once."""
    L = LAYERS[case["layer"]]
    H, I, E, k, T = L["H"], L["I"] // case["tp"], L["E"], L["k"], case["T"]
    active = _active_experts(case)
    elem = 2 if L["fmt"] == "bf16" else 1
    weight_bytes = active * 3.0 * H * I * elem
    if L["fmt"] == "fp8_block":
        weight_bytes += active * 3.0 * (H // 128) * (I // 128) * 4
    elif L["fmt"] == "fp8_channel" or L.get("bias"):
        weight_bytes += active * (2 * I + H) * 4
    routing = T * E * 4 if case["entry"] == "moe" else T * k * 8
    return {"bytes": weight_bytes + T * H * 2 * 2 + routing, "flops": 6.0 * T * k * H * I}


def tolerance(case):
    # bf16 results and a bf16 intermediate; e4m3 layers also round the intermediate to three mantissa bits, where a last
    # bit of the value before it decides between two neighbours
    return {"rel": 1e-2} if LAYERS[case["layer"]]["fmt"] == "bf16" else {"rel": 2e-2}
