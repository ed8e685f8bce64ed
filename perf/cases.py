"""The workloads this package is timed on: routed E8P expert layers and operators, smallest to largest.

Weights, routers and tokens are seeded synthetic data of the distributions the benchmark and the
tests use: uniform codes, scales 0.02 * U(0.5, 1.5), router rows N(0, 0.02^2), tokens N(0, 1).
A model's layers do not find their expert codes in the cache, so a pass over few tokens walks four
layers with weights of their own (each with its own token rows: in a model attention sits between
them), and a pass over many tokens reads more than the cache holds within one layer.
"""

from __future__ import annotations

import torch

from keep_b200 import kernels, moe, router, switch, vq, vq_switch

TOP_K = 6
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
# experts, hidden, inter, scale group along hidden, scale group along inter (0: one scale per row)
SHAPES = {
    "plain": (384, 4096, 2048, 0, 0),        # the benchmark's layer
    "grouped": (192, 5120, 2304, 512, 256),  # the shipped layers: 192 resident experts, group-wise scales
    "pool256": (256, 4096, 2048, 0, 0),      # the pool the sorted-route prefill products are quoted on
}


def listed():
    return [
        # one matrix, one vector: the smallest product a caller of the kernel-level surface makes
        {"name": "qmv_2048x4096", "kind": "qmv", "out": 2048, "in": 4096, "group": 4096, "bits": 16, "dtype": "bf16"},
        # single-stream decode: one token through four layers
        {"name": "decode_1", "kind": "layer", "shape": "plain", "tokens": 1, "layers": 4, "score": "softmax", "dtype": "bf16"},
        # a draft of three tokens verified on layers of the shipped shape and scale groups
        {"name": "grouped_decode_3", "kind": "layer", "shape": "grouped", "tokens": 3, "layers": 4, "score": "sqrtsoftplus", "dtype": "bf16"},
        # routed residency: half the pool resident, the most routed residents with the nested residual
        {"name": "residency_16", "kind": "residency", "tokens": 16, "dtype": "bf16"},
        # 8-bit codes (the operators' default width), enough routes for the sorted strategy
        {"name": "gather_8bit_24", "kind": "gather", "shape": "plain", "tokens": 24, "bits": 8, "dtype": "bf16"},
        # the benchmark's headline batch
        {"name": "decode_64", "kind": "layer", "shape": "plain", "tokens": 64, "layers": 1, "score": "softmax", "dtype": "bf16"},
        # the holder class a model adapter calls, fp16, indices from the model's own router
        {"name": "glu_fp16_96", "kind": "glu", "shape": "pool256", "tokens": 96, "dtype": "fp16"},
        # a full continuous batch of odd size, sigmoid router
        {"name": "decode_251", "kind": "layer", "shape": "plain", "tokens": 251, "layers": 1, "score": "sigmoid", "dtype": "bf16"},
        # a prefill chunk of an ordinary prompt
        {"name": "prefill_1000", "kind": "layer", "shape": "plain", "tokens": 1000, "layers": 1, "score": "softmax", "dtype": "bf16"},
        # the gate projection of a 1024-token prefill through the routed operator, fp16
        {"name": "gather_fp16_1024", "kind": "gather", "shape": "pool256", "tokens": 1024, "bits": 16, "dtype": "fp16"},
        # a ragged prefill chunk on layers of the shipped shape and scale groups
        {"name": "grouped_prefill_1021", "kind": "layer", "shape": "grouped", "tokens": 1021, "layers": 1, "score": "sqrtsoftplus", "dtype": "bf16"},
        # a long prefill chunk
        {"name": "prefill_4096", "kind": "layer", "shape": "plain", "tokens": 4096, "layers": 1, "score": "softmax", "dtype": "bf16"},
    ]


def _log_int(rng, low, high):
    return min(high, int(low * (high / low) ** rng.random() + 0.5))


def draw(rng):
    kind = rng.choice(("layer", "layer", "layer", "layer", "residency", "glu", "gather", "qmv"))
    if kind == "layer":
        shape = rng.choice(("plain", "plain", "grouped"))
        tokens = _log_int(rng, 1, 4096 if shape == "plain" else 1021)
        return {"kind": kind, "shape": shape, "tokens": tokens, "layers": 4 if tokens <= 8 else 1,
                "score": rng.choice(("softmax", "sigmoid", "sqrtsoftplus")), "dtype": rng.choice(("bf16", "bf16", "bf16", "fp16"))}
    if kind == "residency":
        return {"kind": kind, "tokens": _log_int(rng, 1, 256), "dtype": "bf16"}
    if kind == "glu":
        return {"kind": kind, "shape": rng.choice(("pool256", "grouped")), "tokens": _log_int(rng, 1, 512), "dtype": rng.choice(("fp16", "bf16"))}
    if kind == "gather":
        bits = rng.choice((8, 16, 16))
        return {"kind": kind, "shape": rng.choice(("plain", "pool256", "grouped")), "tokens": _log_int(rng, 1, 1024 if bits == 16 else 128), "bits": bits,
                "dtype": rng.choice(("bf16", "fp16"))}
    out, inp = rng.choice(((2048, 4096), (4096, 2048), (2304, 5120), (5120, 2304)))
    return {"kind": kind, "out": out, "in": inp, "group": rng.choice((256, inp)), "bits": rng.choice((8, 16, 16)), "dtype": rng.choice(("bf16", "fp16", "fp32"))}


# ---- inputs ------------------------------------------------------------------------------------

def _codes(gen, shape, bits):
    if bits == 8:
        return torch.randint(0, 256, shape, generator=gen, device="cuda", dtype=torch.uint8)
    return torch.randint(-32768, 32768, shape, generator=gen, device="cuda", dtype=torch.int16).view(torch.uint16)


def _scales(gen, shape):
    return (0.02 * (0.5 + torch.rand(shape, generator=gen, device="cuda"))).to(torch.float16)


def _matrix(gen, experts, out, inp, group, bits=16):
    return _codes(gen, (experts, out, inp // 8), bits), _scales(gen, (experts, out, inp // (group or inp)))


def _experts(gen, shape):
    experts, hidden, inter, gh, gi = SHAPES[shape]
    return _matrix(gen, experts, inter, hidden, gh), _matrix(gen, experts, inter, hidden, gh), _matrix(gen, experts, hidden, inter, gi)


def _normal(gen, shape, dtype):
    return torch.randn(shape, generator=gen, device="cuda").to(dtype)


def _picks(gen, tokens, experts):
    return torch.rand((tokens, experts), generator=gen, device="cuda").topk(TOP_K, dim=1).indices.to(torch.int32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    if kind == "layer":
        experts, hidden = SHAPES[case["shape"]][:2]
        layers, xs = [], []
        for _ in range(case["layers"]):
            w1, w3, w2 = (moe.Projection(*w) for w in _experts(gen, case["shape"]))
            gate = _normal(gen, (experts, hidden), torch.float32).mul_(0.02).to(torch.bfloat16)
            extra = {"route_scale": 1.5, "swiglu_limit": 10.0} if case["score"] == "sqrtsoftplus" else {}
            layers.append(moe.RoutedMoELayer(gate, w1, w3, w2, top_k=TOP_K, score_func=case["score"], **extra))
            xs.append(_normal(gen, (case["tokens"], hidden), dtype))
        return {"kind": kind, "layers": layers, "xs": xs}
    if kind == "residency":
        pool, hidden, inter = SHAPES["plain"][:3]
        resident, hot = pool // 2, 32
        gate = _normal(gen, (pool, hidden), torch.float32).mul_(0.02).to(torch.bfloat16)
        there = torch.randperm(pool, generator=gen, device="cuda")[:resident].sort().values
        slot_of = torch.full((pool,), -1, dtype=torch.int32, device="cuda")
        slot_of[there] = torch.arange(resident, dtype=torch.int32, device="cuda")
        bias = torch.full((pool,), router.OFF, device="cuda")
        bias[there] = 0.0
        picks = router.routed_topk(_normal(gen, (1024, hidden), dtype), gate, bias, None, slot_of, top_k=TOP_K).served_slot
        hot_slots = torch.bincount(picks.reshape(-1).clamp(min=0), minlength=resident).topk(hot).indices
        hot_of_slot = torch.full((resident,), -1, dtype=torch.int32, device="cuda")
        hot_of_slot[hot_slots] = torch.arange(hot, dtype=torch.int32, device="cuda")

        def tiered(out, inp):
            return moe.Projection(*_matrix(gen, resident, out, inp, 0), _codes(gen, (hot, out, inp // 8), 8),
                                  torch.full((hot, out, 1), 0.005, dtype=torch.float16, device="cuda"))

        layer = moe.RoutedMoELayer(gate, tiered(inter, hidden), tiered(inter, hidden), tiered(hidden, inter), top_k=TOP_K, tau=0.3,
                                   served_bias=bias, slot_of=slot_of, hot_of_slot=hot_of_slot)
        return {"kind": "layer", "layers": [layer], "xs": [_normal(gen, (case["tokens"], hidden), dtype)]}
    if kind == "glu":
        experts, hidden, inter, gh, gi = SHAPES[case["shape"]]
        w1, w3, w2 = _experts(gen, case["shape"])

        def linear(w, out, inp, group):
            return switch.QuantizedVQSwitchLinear(input_dims=inp, output_dims=out, num_experts=experts, codes=w[0], scales=w[1],
                                                  group_size=group or inp, code_bits=16, use_gather_vqmm=True, route_strategy="auto")

        glu = switch.QuantizedVQSwitchGLU(gate_proj=linear(w1, inter, hidden, gh), up_proj=linear(w3, inter, hidden, gh), down_proj=linear(w2, hidden, inter, gi))
        return {"kind": kind, "glu": glu, "x": _normal(gen, (case["tokens"], hidden), dtype), "picks": _picks(gen, case["tokens"], experts)}
    if kind == "gather":
        experts, hidden, inter, gh, _ = SHAPES[case["shape"]]
        codes, scales = _matrix(gen, experts, inter, hidden, gh, case["bits"])
        return {"kind": kind, "args": (_normal(gen, (case["tokens"], hidden), dtype), codes, scales,
                                       vq.table_on(codes.device, "e8p" if case["bits"] == 16 else "e8_1bit"), _picks(gen, case["tokens"], experts)),
                "named": dict(input_dims=hidden, output_dims=inter, group_size=gh or hidden, code_bits=case["bits"])}
    codes, scales = _matrix(gen, 1, case["out"], case["in"], case["group"], case["bits"])
    return {"kind": kind, "args": (_normal(gen, (case["in"],), dtype), codes[0], scales[0], vq.table_on(codes.device, "e8p" if case["bits"] == 16 else "e8_1bit")),
            "named": dict(in_dim=case["in"], out_dim=case["out"], group_size=case["group"], code_bits=case["bits"])}


def run(state):
    kind = state["kind"]
    if kind == "layer":
        done = []
        for layer, x in zip(state["layers"], state["xs"]):
            y, r = layer.decode(x)
            done.append({"y": y, "served": r.served_expert, "weight": r.served_weight, "want": r.want, "admit": r.admit})
        return done
    if kind == "glu":
        return state["glu"](state["x"], state["picks"])
    if kind == "gather":
        return vq_switch.gather_vqmm(*state["args"], **state["named"])
    return kernels.vq_qmv(*state["args"], **state["named"])


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    kind, wide = case["kind"], 4 if case["dtype"] == "fp32" else 2
    if kind == "qmv":
        out, inp = case["out"], case["in"]
        return {"bytes": out * inp // 8 * case["bits"] // 8 + out * (inp // case["group"]) * 2 + (inp + out) * wide, "flops": 2 * out * inp}
    tokens, routes = case["tokens"], case["tokens"] * TOP_K
    experts, hidden, inter, gh, gi = SHAPES["plain" if kind == "residency" else case["shape"]]
    touch = lambda n: n * (1.0 - (1.0 - TOP_K / n) ** tokens)  # noqa: E731 - experts that uniform routing touches
    matrix = hidden * inter / 8
    if kind == "gather":
        return {"bytes": touch(experts) * (matrix * case["bits"] / 8 + inter * hidden / (gh or hidden) * 2) + (tokens * hidden + routes * inter) * wide,
                "flops": 2 * routes * hidden * inter}
    scales = 2 * (2 * inter * hidden / (gh or hidden) + hidden * inter / (gi or inter))
    if kind == "glu":
        return {"bytes": touch(experts) * (6 * matrix + scales) + (tokens + routes) * hidden * wide, "flops": 6 * routes * hidden * inter}
    gate = experts * hidden * 2
    io = 2 * tokens * hidden * wide + routes * 20
    if kind == "residency":
        used = touch(experts // 2)
        return {"bytes": used * (6 * matrix + scales) + used / 6 * (3 * matrix + scales) + gate + io, "flops": routes * 6 * hidden * inter + 2 * tokens * experts * hidden}
    return {"bytes": case["layers"] * (touch(experts) * (6 * matrix + scales) + gate + io), "flops": case["layers"] * (routes * 6 * hidden * inter + 2 * tokens * experts * hidden)}


def tolerance(case):
    # Four times the distance (2-norm) of the present kernels from the same path in 64 bits, measured on
    # the listed cases, is 1.5e-2 / 1.8e-3 for a bf16 / fp16 layer (three roundings to the activation
    # dtype), 6.6e-3 / 8.5e-4 / 1.2e-6 for one product; expert picks were equal in every case.
    if case["kind"] in ("layer", "residency", "glu"):
        return {"rel": {"bf16": 1e-2, "fp16": 1.8e-3}[case["dtype"]], "differ": 1e-3}
    return {"rel": {"bf16": 6.6e-3, "fp16": 8.5e-4, "fp32": 1.2e-6}[case["dtype"]]}
