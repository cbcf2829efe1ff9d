"""Workloads by which the speed of this package is judged: what a program that uses it has it do, over the range of
sizes, weight formats and options that its configurations, tests and benchmark name.

A case is a dict of plain values.  ``kind`` names the way in:

* ``layer``   :class:`MoELayer` prefill, called eagerly (router, grouping, quantise, both contractions, combine)
* ``graph``   the same layer on a decode batch, captured once and replayed for every token, as a serving loop does
* ``cte``     prefill through the drop-in calls ``router_topk`` -> ``moe_group_tokens`` -> ``moe_cte``
* ``tkg``     decode through ``router_topk`` -> ``moe_tkg`` (each token through its own top-k experts)
* ``block``   decode through ``moe_block_tkg``: RMSNorm + residual, router, every local expert on every token

``weights`` is the element type of the expert weights: ``e4m3`` / ``e5m2`` (MXFP8), ``e2m1`` (MXFP4), ``bf16``, or
``fp8row`` (fp8 with one factor per output row).  ``x4`` says that the weights come from the reference's packed
storage, whose hidden axis the activation quantiser has to follow.  Weights are prepared once, as a program does when
it loads a model; hidden states, routing and outputs belong to the pass.
"""

import math

import torch

import nki_library_b200 as moe
from nki_library_b200.layer import MoELayer, random_expert_weights
from nki_library_b200.weights import prepare_dense

MX_CODES = {"e4m3": 0, "e5m2": 1, "e2m1": 5}
WEIGHT_BYTES = {"e4m3": 1 + 1 / 32, "e5m2": 1 + 1 / 32, "e2m1": 0.5 + 1 / 32, "bf16": 2.0, "fp8row": 1.0}


def _case(kind, T, H, I, E, K, B=128, weights="e4m3", x4=False, zipf=0.0, local=0, act="SiLU", bias=False, clamp=0.0):
    return dict(kind=kind, T=T, H=H, I=I, E=E, K=K, B=B, weights=weights, x4=x4, zipf=zipf, local=local, act=act,
                bias=bias, clamp=clamp)


def listed():
    cases = {
        # the smallest layer of the tests and the smoke run: launches and host work
        "prefill-tiny": _case("layer", 256, 512, 1024, 4, 2),
        # the benchmark's headline: a Mixtral-8x7B-shaped prefill of 4096 tokens
        "prefill-mixtral": _case("layer", 4096, 4096, 14336, 8, 2, B=512),
        # many small experts with a skewed load: most blocks are padded or partly filled
        "prefill-finegrained": _case("layer", 8192, 7168, 2048, 256, 8, zipf=1.2),
        # the largest batch: 32768 tokens over 128 experts, through the drop-in calls
        "prefill-32768": _case("cte", 32768, 4096, 1536, 128, 8, B=256),
        # a ragged prompt on weights in the reference's storage, with biases, clamps and the Swish activation
        "prefill-ragged": _case("cte", 2531, 3072, 1536, 64, 4, B=256, x4=True, act="Swish", bias=True, clamp=7.0),
        # a non-MX model: bf16 weights on the dense kernels
        "prefill-bf16": _case("cte", 1800, 2048, 4096, 8, 2, B=256, weights="bf16", act="GELU"),
        # decode of a batch of 64 sequences, weight streaming
        "decode-mixtral": _case("tkg", 64, 4096, 14336, 8, 2),
        # the same with 4-bit weights
        "decode-mxfp4": _case("tkg", 64, 4096, 14336, 8, 2, weights="e2m1"),
        # a handful of sequences on many experts: latency
        "decode-few": _case("tkg", 3, 3072, 1536, 128, 8, x4=True),
        # a serving loop's captured step
        "decode-graph": _case("graph", 16, 4096, 1536, 128, 8),
        # the whole decode block on one rank's 16 of 128 experts, every token through every one of them
        "decode-block": _case("block", 128, 3072, 1536, 128, 4, x4=True, local=16),
        # decode on fp8 weights with per-row factors
        "decode-fp8row": _case("tkg", 32, 4096, 1536, 16, 2, weights="fp8row", bias=True),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges: batch sizes over their logarithm, hidden and intermediate sizes in the steps
    that the formats allow, weights of at most 4 GB and at most the arithmetic of the larger prefill cases."""
    while True:
        kind = rng.choice(["layer", "cte", "cte", "tkg", "tkg", "graph", "block"])
        x4 = kind in ("cte", "tkg", "block") and rng.random() < 0.5
        weights = rng.choice(["e4m3", "e4m3", "e5m2", "e2m1"])
        if kind in ("cte", "tkg") and rng.random() < 0.3:
            weights, x4 = rng.choice(["bf16", "fp8row"]), False
        step = 512 if x4 else 128
        H = step * _log_int(rng, max(1, 512 // step), 7168 // step)
        I = step * _log_int(rng, max(1, 256 // step), 14336 // step)
        if not x4 and weights not in ("e2m1",) and I > 256 and rng.random() < 0.3:
            I -= 32 * rng.randint(1, 3)
        E = _log_int(rng, 4, 256)
        K = min(rng.randint(1, 8), E)
        T = _log_int(rng, 200, 32768) if kind in ("layer", "cte") else _log_int(rng, 1, 128)
        B = rng.choice([128, 256, 512]) if kind in ("layer", "cte") else 128
        local = 0
        if kind == "block":
            E = 8 * max(1, E // 8)
            K = min(K, E)
            local = E // 8
        case = _case(kind, T, H, I, E, K, B, weights, x4, rng.choice([0.0, 0.0, 1.2]), local,
                     rng.choice(["SiLU", "SiLU", "Swish", "GELU", "GELU_Tanh_Approx"]),
                     kind in ("cte", "tkg") and rng.random() < 0.3, 0.0)
        held = 3.0 * (local or E) * H * I * WEIGHT_BYTES[weights]
        if held <= 4e9 and work(case)["flops"] <= 4e12:
            return case


# ------------------------------------------------------------------ what a program has in hand before the call
def _x4_weights(case, E, gen):
    """Expert weights in the reference's x4-packed storage: element codes of values that fill the element type's range
    the way a quantised Gaussian does, block scales around those of weights ~N(0, 0.02)."""
    H, I, nt = case["H"], case["I"], case["H"] // 512
    p_i, n_i = (128, I // 512) if I > 512 else (I // 4, 1)

    def codes(*shape):
        if case["weights"] == "e2m1":
            return torch.randint(0, 256, (*shape, 2), dtype=torch.uint8, device="cuda", generator=gen).view(torch.int16)[..., 0]
        dt = torch.float8_e5m2 if case["weights"] == "e5m2" else torch.float8_e4m3fn
        return (torch.randn((*shape, 4), device="cuda", generator=gen) * 100).clamp(-448, 448).to(dt).view(torch.int32)[..., 0]

    base = 121 if case["weights"] == "e2m1" else 114  # 2^-6 x (values of about 2) or 2^-13 x (values of about 100)

    def scales(*shape):
        return torch.randint(base - 1, base + 2, shape, dtype=torch.uint8, device="cuda", generator=gen)

    b_gu = b_d = None
    if case["bias"]:
        b_gu = torch.randn((E, p_i, 2, n_i, 4), device="cuda", generator=gen) * 0.1
        b_d = torch.randn((E, H), device="cuda", generator=gen) * 0.1
    return moe.prepare_from_nki(codes(E, 128, 2, nt, I), scales(E, 16, 2, nt, I), codes(E, p_i, n_i, H),
                                scales(E, p_i // 8, n_i, H), b_gu, b_d, w_format=case["weights"])


def _dense_weights(case, E, gen):
    H, I = case["H"], case["I"]

    def tensor(*shape):
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        for e in range(E):
            t[e] = torch.randn(shape[1:], device="cuda", generator=gen) * 0.02
        return t

    w1, w2 = tensor(E, H, 2, I), tensor(E, I, H)
    b_gu = b_d = s1 = s2 = None
    if case["bias"]:
        b_gu = torch.randn((E, 2, I), device="cuda", generator=gen) * 0.1
        b_d = torch.randn((E, H), device="cuda", generator=gen) * 0.1
    if case["weights"] == "fp8row":
        w1, w2 = ((w * 5000).clamp(-448, 448).to(torch.float8_e4m3fn) for w in (w1, w2))
        s1 = (torch.rand((E, 2, I), device="cuda", generator=gen) + 0.5) / 5000
        s2 = (torch.rand((E, H), device="cuda", generator=gen) + 0.5) / 5000
    return prepare_dense(w1, w2, b_gu, b_d, s1, s2)


def _weights(case, gen, seed):
    E = case["local"] or case["E"]
    if case["weights"] in ("bf16", "fp8row"):
        return _dense_weights(case, E, gen)
    if case["x4"]:
        return _x4_weights(case, E, gen)
    w = random_expert_weights(E, case["H"], case["I"], "cuda", seed=seed, w_format=MX_CODES[case["weights"]])
    if case["bias"]:
        w.bias_gu = torch.randn((E, 2 * case["I"]), device="cuda", generator=gen) * 0.1
        w.bias_d = torch.randn((E, case["H"]), device="cuda", generator=gen) * 0.1
    return w


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    T, H, E, K, B = (case[k] for k in "THEKB")
    weights = _weights(case, gen, seed)
    hidden = torch.randn((T, H), device="cuda", generator=gen).to(torch.bfloat16)
    router_w = (torch.randn((H, E), device="cuda", generator=gen) * 0.02).to(torch.bfloat16)
    router_b = None
    if case["zipf"]:
        rank = torch.randperm(E, device="cuda", generator=gen).float() + 1.0
        router_b = (-case["zipf"] * torch.log(rank)).to(torch.bfloat16)
    state = dict(case=case, weights=weights, hidden=hidden, router_w=router_w, router_b=router_b)
    if case["kind"] in ("layer", "graph"):
        layer = MoELayer(router_w, weights, K, B, T, router_bias=router_b, act_fn=moe.ActFnType[case["act"]])
        state["layer"] = layer
        if case["kind"] == "graph":
            layer.forward(hidden)
            torch.cuda.synchronize()
            layer.capture(hidden)
    elif case["kind"] == "block":
        state["residual"] = torch.randn((T, H), device="cuda", generator=gen).to(torch.bfloat16)
        state["gamma"] = (torch.randn((H,), device="cuda", generator=gen) * 0.1 + 1.0).to(torch.bfloat16)
        state["rank_id"] = torch.full((1, 1), 1 if E > case["local"] else 0, dtype=torch.int32, device="cuda")
    else:  # router_topk writes into tensors of its caller
        state["logits"] = torch.empty((T, E), device="cuda")
        state["aff"] = torch.empty((T, E), device="cuda")
        state["idx"] = torch.empty((T, K), dtype=torch.int32, device="cuda")
        state["n_blocks"] = moe.get_n_blocks(T, K, E, B)
    return state


# ------------------------------------------------------------------ one pass
def _route(s):
    moe.router_topk(s["hidden"], s["router_w"], s["router_b"], s["logits"], s["aff"], s["idx"],
                    moe.RouterActFnType.SOFTMAX, s["case"]["K"], 1, 0, norm_topk_prob=True)


def run(state):
    case = state["case"]
    kind, act = case["kind"], moe.ActFnType[case["act"]]
    hi = case["clamp"] or None
    if kind == "layer":
        layer = state["layer"]
        out = layer.forward(state["hidden"])
        return {"out": out, "index": layer.idx, "affinities": layer.aff}
    if kind == "graph":
        layer = state["layer"]
        out = layer.replay()
        return {"out": out, "index": layer.idx, "affinities": layer.aff}
    if kind == "block":
        out, logits, residual = moe.moe_block_tkg(
            state["hidden"], state["gamma"], state["router_w"], state["weights"], None, router_bias=state["router_b"],
            top_k=case["K"], router_act_fn=moe.RouterActFnType.SOFTMAX, norm_topk_prob=True,
            expert_affinities_scaling_mode=moe.ExpertAffinityScaleMode.POST_SCALE, hidden_act_fn=act,
            is_all_expert=True, rank_id=state["rank_id"], residual=state["residual"])
        return {"out": out, "logits": logits, "residual": residual}
    _route(state)
    if kind == "tkg":
        out = moe.moe_tkg(
            state["hidden"], state["weights"], None, state["aff"], state["idx"], False,
            expert_affinities_scaling_mode=moe.ExpertAffinityScaleMode.POST_SCALE, activation_fn=act,
            gate_clamp_upper_limit=hi, up_clamp_upper_limit=hi, up_clamp_lower_limit=-hi if hi else None)
    else:
        dense = case["weights"] in ("bf16", "fp8row")
        g = moe.moe_group_tokens(state["idx"], case["E"], case["B"], state["n_blocks"])
        impl = moe.MoECTEImplementation
        out = moe.moe_cte(
            state["hidden"], state["aff"].view(-1, 1), state["weights"], None, g["token_position_to_id"],
            g["block_to_expert"], case["B"], moe.MoECTESpec(impl.shard_on_i_hybrid if dense else impl.shard_on_block_mx),
            conditions=g["conditions"], activation_function=act, skip_dma=moe.SkipMode(True, False),
            gate_clamp_upper_limit=hi, up_clamp_upper_limit=hi, up_clamp_lower_limit=-hi if hi else None)
    return {"out": out, "index": state["idx"], "affinities": state["aff"], "logits": state["logits"]}


# ------------------------------------------------------------------ what it cannot do without
def work(case):
    T, H, I, E, K = (case[k] for k in "THIEK")
    if case["kind"] == "block":
        pairs, active = T * case["local"], case["local"]
    else:
        # expected number of experts that at least one token chose, under even routing
        pairs, active = T * K, E * (1.0 - (1.0 - K / E) ** T)
    expert = 3.0 * H * I * WEIGHT_BYTES[case["weights"]]
    rows = 4 if case["kind"] == "block" else 2  # hidden in and out; the block also takes and returns the residual
    return {"bytes": active * expert + rows * T * H * 2 + H * E * 2 + T * E * 4 + T * K * 4,
            "flops": 6.0 * pairs * H * I + 2.0 * T * H * E}


def tolerance(case):
    # Outputs are sums of rows that are rounded to bf16 one by one and once more at the end (each rounding: 1.7e-3 of
    # the norm), behind an MXFP8 re-quantisation whose ties may fall to either side when the fp32 sums before it are
    # taken in another order (measured against the CUDA-core kernels: up to 5e-4 of the norm, single values off by up
    # to 0.03 of the rms); expert ids may differ where two logits tie.
    return {"rel": 1e-2, "max": 0.2, "differ": 1e-3}
