"""The framework's work as a program that serves the two models has it done, case by case, through the
public entry points: quantised linear layers, the dense MLP chain of the 31B model, the MoE layer and the
feed-forward block of the 26B model, and the weight formats a loader works with.

A case is a dict of plain values:
  op       linear / mlp / moe / ffn / weights
  storage  of the weights: nvfp4, fp8 or bf16
  rows     token rows of the pass: 1 .. 64 in a decode step, up to 4096 (MoE: 8192) in a prefill chunk
Weights are N(0, 0.02) and activations N(0, 1), as in the benchmark configurations.
"""
from __future__ import annotations

import math

import torch

import gewell_b200 as gw
from gewell_b200 import _lib

HIDDEN, INTER, EXPERTS, TOPK = 2816, 704, 128, 8        # the 26B model's MoE
SHARED = 2112                                           # its shared MLP
HIDDEN31, MLP31 = 5376, 21504                           # the 31B model

# bytes of a weight matrix element (NVFP4: half a byte and one scale byte for sixteen elements)
WEIGHT_BYTES = {"nvfp4": 0.5625, "fp8": 1.0, "bf16": 2.0}
# what one floating-point operation of a kind takes, in units of an FP4 one
RATE = {"nvfp4": 1.0, "fp8": 2.0, "bf16": 4.0}
# (K, N) of the projections of both models
PROJECTIONS = [(2816, 2816), (2816, 4096), (2816, 8192), (4096, 2816), (8192, 2816), (5376, 2048), (5376, 4096), (5376, 8192),
               (5376, 16384), (8192, 5376), (16384, 5376), (5376, 21504), (21504, 5376), (5376, 43008)]


def listed():
    return [
        # a small projection at a small decode batch: launches and latency
        {"name": "linear nvfp4 16x2816x2816", "op": "linear", "storage": "nvfp4", "rows": 16, "k": 2816, "n": 2816},
        # the joined gate/up projection of the 31B model in a decode step of eight sequences
        {"name": "linear fp8 8x5376x43008", "op": "linear", "storage": "fp8", "rows": 8, "k": 5376, "n": 43008, "channel": True},
        # the joined Q|K|V projection over a ragged prefill chunk
        {"name": "linear fp8 1025x5376x16384", "op": "linear", "storage": "fp8", "rows": 1025, "k": 5376, "n": 16384, "channel": True},
        # the 31B down projection over a full prefill chunk
        {"name": "linear nvfp4 4096x21504x5376", "op": "linear", "storage": "nvfp4", "rows": 4096, "k": 21504, "n": 5376},
        # an unquantised projection of the 26B model over a short prompt
        {"name": "linear bf16 200x2816x8192", "op": "linear", "storage": "bf16", "rows": 200, "k": 2816, "n": 8192},
        # one layer's MLP of the 31B model for a single sequence, FP4 activations
        {"name": "mlp nvfp4 decode 1", "op": "mlp", "storage": "nvfp4", "rows": 1, "hidden": HIDDEN31, "mlp": MLP31,
         "policy": "always", "phase": "decode"},
        # the same where the policy keeps decode activations in BF16
        {"name": "mlp nvfp4 w4a16 decode 5", "op": "mlp", "storage": "nvfp4", "rows": 5, "hidden": HIDDEN31, "mlp": MLP31,
         "policy": "prefill", "phase": "decode"},
        # FP8 weights, a prefill chunk (the largest case by time)
        {"name": "mlp fp8 prefill 2048", "op": "mlp", "storage": "fp8", "rows": 2048, "hidden": HIDDEN31, "mlp": MLP31,
         "policy": "always", "phase": "prefill"},
        # the MoE layer in a decode step of 64 sequences: nearly every expert is touched by a few rows
        {"name": "moe nvfp4 64", "op": "moe", "storage": "nvfp4", "rows": 64, "fp4": True, "skew": 0.0, "scales": "layer"},
        # a ragged prompt whose routing prefers some experts, experts calibrated one by one
        {"name": "moe nvfp4 777 skewed", "op": "moe", "storage": "nvfp4", "rows": 777, "fp4": True, "skew": 1.2, "scales": "expert"},
        # the MoE layer over a large prefill batch
        {"name": "moe nvfp4 8192", "op": "moe", "storage": "nvfp4", "rows": 8192, "fp4": True, "skew": 0.0, "scales": "layer"},
        # the whole feed-forward block of a 26B layer in a decode step of eight sequences
        {"name": "ffn nvfp4 decode 8", "op": "ffn", "storage": "nvfp4", "rows": 8, "policy": "always", "phase": "decode"},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choices(["linear", "mlp", "moe", "ffn", "weights"], [35, 20, 25, 12, 8])[0]
    storage = rng.choices(["nvfp4", "fp8", "bf16"], [60, 25, 15])[0]
    rows = _log_uniform(rng, 1, 4096)
    if op == "linear":
        k, n = rng.choice(PROJECTIONS)
        if rng.random() < 0.3:         # another model's widths: any that the storage allows
            step_k, step_n = {"nvfp4": (64, 128), "fp8": (16, 16), "bf16": (8, 8)}[storage]
            k, n = (max(1, _log_uniform(rng, 512, 8192) // s) * s for s in (step_k, step_n))
        case = {"op": op, "storage": storage, "rows": _capped(rows, 2.0 * k * n, storage), "k": k, "n": n}
        if storage == "fp8":
            case["channel"] = rng.random() < 0.5
        return case
    if op == "mlp":
        hidden, mlp = HIDDEN31, MLP31
        if rng.random() < 0.3:
            hidden, mlp = 128 * rng.randint(8, 40), 128 * rng.randint(16, 120)
        rows = _capped(rows, 6.0 * hidden * mlp, storage)
        return {"op": op, "storage": storage, "rows": rows, "hidden": hidden, "mlp": mlp, "policy": rng.choice(["always", "prefill"]),
                "phase": "decode" if rows <= 64 else "prefill"}
    if op == "moe":
        fp4 = storage != "nvfp4" or rng.random() < 0.8
        rows = _log_uniform(rng, 1, 8192) if storage == "nvfp4" and fp4 else rows
        return {"op": op, "storage": storage, "rows": rows, "fp4": fp4, "skew": rng.choice([0.0, 0.0, 1.2]),
                "scales": rng.choice(["layer", "expert"])}
    if op == "ffn":
        return {"op": op, "storage": storage, "rows": rows, "policy": rng.choice(["always", "prefill"]),
                "phase": "decode" if rows <= 64 else "prefill"}
    what = rng.choice(["pack", "dequantize", "qdq"])
    # the three formats of a weight matrix on its way to or from the device; N rows as a joined or single projection has them
    return {"op": op, "storage": "nvfp4" if what == "dequantize" else rng.choice(["nvfp4", "fp8"]), "what": what,
            "n": 128 * rng.randint(6, 168), "k": 64 * rng.randint(11, 84)}


def _capped(rows, flops_per_row, storage):
    """Rows of a drawn case, so that it takes no longer than the largest listed one."""
    limit = 6.0 * HIDDEN31 * MLP31 * 2048 * RATE["fp8"]
    return max(1, min(rows, int(limit / (flops_per_row * RATE[storage]))))


# --------------------------------------------------------------------------- what a program has in hand

def _normal(g, shape, std=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * std).bfloat16()


def _weight(g, storage, n, k, input_scale, channel=False):
    """One bound matrix [n, k]."""
    w = _normal(g, (n, k), 0.02)
    if storage == "bf16":
        return w
    if storage == "nvfp4":
        return gw.nvfp4_pack_weights(w, input_scale)
    if channel:
        row_scale = (w.float().abs().amax(dim=1) / 448).contiguous()
        return gw.Fp8Weight(gw.fp8_pack_weights(w, 0.0, row_scale), input_scale, 1.0, (row_scale * input_scale).contiguous())
    scale = float(w.float().abs().max() / 448)
    return gw.Fp8Weight(gw.fp8_pack_weights(w, scale), input_scale, scale)


def _input_scale(storage, amax=6.0):
    return amax / (448.0 if storage == "fp8" else 2688.0)


def _halves(weight, storage, n, k):
    """The two matrices of a joined pair [2n, k], as the loader leaves them: back to back."""
    if storage == "bf16":
        return weight[:n], weight[n:]
    if storage == "fp8":
        return tuple(gw.Fp8Weight(weight.data[s], weight.input_scale, weight.weight_scale, weight.channel_scales[s])
                     for s in (slice(0, n), slice(n, 2 * n)))
    split = gw.nvfp4_scale_storage_bytes(n, k)
    return (gw.Nvfp4Weight(weight.data[:n], weight.scales[:split], weight.input_scale, weight.weight_scale),
            gw.Nvfp4Weight(weight.data[n:], weight.scales[split:], weight.input_scale, weight.weight_scale))


def _expert_matrices(g, storage, n, k, scales):
    """One matrix of every expert; scales[e] is the expert's input scale."""
    padded = (n + 127) // 128 * 128 if storage == "nvfp4" else n
    w = torch.zeros((EXPERTS, padded, k), dtype=torch.bfloat16, device="cuda")
    w[:, :n] = torch.randn((EXPERTS, n, k), generator=g, device="cuda").mul_(0.02)
    if storage == "bf16":
        return list(w)
    if storage == "fp8":
        scale = float(w.abs().max()) / 448
        data = gw.fp8_pack_weights(w.view(-1, k), scale).view(EXPERTS, padded, k)
        return [gw.Fp8Weight(data[e], scales[e], scale) for e in range(EXPERTS)]
    packed = gw.nvfp4_pack_weights(w.view(-1, k))
    data, tiles = packed.data.view(EXPERTS, padded, k // 2), packed.scales.view(EXPERTS, -1)
    return [gw.Nvfp4Weight(data[e], tiles[e], scales[e], packed.weight_scale) for e in range(EXPERTS)]


def _experts(g, storage, per_expert_scales):
    first = [_input_scale(storage) * (1.0 + (e % 16) / 64.0 if per_expert_scales else 1.0) for e in range(EXPERTS)]
    down = [_input_scale(storage, 16.0)] * EXPERTS
    gate = _expert_matrices(g, storage, INTER, HIDDEN, first)
    up = _expert_matrices(g, storage, INTER, HIDDEN, first)
    return gw.ExpertTable(list(zip(gate, up, _expert_matrices(g, storage, HIDDEN, INTER, down))))


def _flags(storage):
    return {"has_bf16": storage == "bf16", "has_fp8": storage == "fp8", "has_nvfp4": storage == "nvfp4"}


def _prepare_linear(case, g):
    rows, k, n, storage = case["rows"], case["k"], case["n"], case["storage"]
    weight = _weight(g, storage, n, k, _input_scale(storage), case.get("channel", False))
    if storage == "nvfp4":
        plan = gw.Nvfp4Plan(rows, k, n)
    elif storage == "fp8":
        plan = gw.Fp8Plan(rows, k, n, case["channel"])
    else:
        plan = gw.Bf16Plan(rows, k, n)
    return {"plan": plan, "weight": weight, "x": _normal(g, (rows, k)),
            "y": torch.empty((rows, n), dtype=torch.bfloat16, device="cuda"),
            "scratch": torch.empty(max(256, plan.scratch_bytes()), dtype=torch.uint8, device="cuda")}


def _prepare_mlp(case, g):
    rows, hidden, mlp, storage = case["rows"], case["hidden"], case["mlp"], case["storage"]
    both = _weight(g, storage, 2 * mlp, hidden, _input_scale(storage), channel=True)
    gate, up = _halves(both, storage, mlp, hidden)
    down = _weight(g, storage, hidden, mlp, _input_scale(storage, 32.0))
    chain = gw.MlpChain(hidden, mlp, max(64, rows), getattr(_lib, "POLICY_" + case["policy"].upper()))
    chain.prepare(rows)
    bound = [gw.make_projection(w, i, o) for w, i, o in ((gate, hidden, mlp), (up, hidden, mlp), (down, mlp, hidden))]
    return {"chain": chain, "bound": bound, "keep": (both, down), "x": _normal(g, (rows, hidden)),
            "phase": getattr(_lib, "PHASE_" + case["phase"].upper())}


def _prepare_moe(case, g):
    rows, storage = case["rows"], case["storage"]
    table = _experts(g, storage, case["scales"] == "expert")
    if storage == "nvfp4" and not case["fp4"]:
        table.enable_w4a16()
    logits = torch.randn((rows, EXPERTS), generator=g, device="cuda")
    if case["skew"]:                   # expert popularity by a power law, the experts in an order of their own
        order = torch.randperm(EXPERTS, generator=g, device="cuda") + 1
        logits = logits - case["skew"] * order.float().log()
    return {"workspace": gw.MoeWorkspace(max(64, rows), fp8_experts=storage == "fp8"), "table": table, "rows": rows,
            "flags": _flags(storage), "fp4": case["fp4"], "x": _normal(g, (rows, HIDDEN)), "scores": logits.bfloat16(),
            "expert_scales": torch.ones(EXPERTS, dtype=torch.bfloat16, device="cuda"),
            "y": torch.empty((rows, HIDDEN), dtype=torch.bfloat16, device="cuda")}


def _prepare_ffn(case, g):
    rows, storage = case["rows"], case["storage"]
    table = _experts(g, storage, False)
    if storage == "nvfp4" and case["policy"] == "prefill":
        table.enable_w4a16()

    def shared(n, k, amax):
        weight = _weight(g, storage, n, k, _input_scale(storage, amax))
        if storage == "nvfp4" and n % 128:
            data = torch.zeros(((n + 127) // 128 * 128, k // 2), dtype=torch.uint8, device="cuda")
            data[:n] = weight.data
            weight = gw.Nvfp4Weight(data, weight.scales, weight.input_scale, weight.weight_scale)
        return weight

    def norm():
        return 1.0 + 0.25 * _normal(g, (HIDDEN,))

    layer = {"pre_feedforward_norm": norm(), "router_scale": norm(), "pre_feedforward_norm_2": norm(),
             "post_feedforward_norm_1": norm(), "post_feedforward_norm_2": norm(), "post_feedforward_norm": norm(),
             "layer_scalar": torch.tensor([0.8203125], dtype=torch.bfloat16, device="cuda"),
             "router_proj": _normal(g, (EXPERTS, HIDDEN)),
             "router_per_expert_scale": torch.ones(EXPERTS, dtype=torch.bfloat16, device="cuda"),
             "gate": shared(SHARED, HIDDEN, 6.0), "up": shared(SHARED, HIDDEN, 6.0), "down": shared(HIDDEN, SHARED, 16.0),
             "experts": table, **_flags(storage)}
    block = gw.FfnBlock([layer], max(64, rows), getattr(_lib, "POLICY_" + case["policy"].upper()), fp8_experts=storage == "fp8")
    block.prepare(rows, getattr(_lib, "PHASE_" + case["phase"].upper()))
    source = _normal(g, (rows, HIDDEN), 2.0)
    return {"block": block, "layer": layer, "source": source, "hidden": torch.empty_like(source)}


def _prepare_weights(case, g):
    w = _normal(g, (case["n"], case["k"]), 0.02)
    if case["what"] == "dequantize":
        return {"what": case["what"], "packed": gw.nvfp4_pack_weights(w), "n": case["n"], "k": case["k"], "out": w}
    return {"what": case["what"], "storage": case["storage"], "w": w,
            "scale": float(w.float().abs().max() / 448) if case["storage"] == "fp8" else None}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    state = {"linear": _prepare_linear, "mlp": _prepare_mlp, "moe": _prepare_moe, "ffn": _prepare_ffn,
             "weights": _prepare_weights}[case["op"]](case, g)
    state["op"] = case["op"]
    return state


# --------------------------------------------------------------------------- one pass

def run(state):
    op = state["op"]
    if op == "linear":
        return state["plan"].run(state["x"], state["weight"], state["y"], state["scratch"])
    if op == "mlp":
        gate, up, down = state["bound"]
        return state["chain"].run(gate, up, down, state["x"], state["phase"])
    if op == "moe":
        return state["workspace"].run(state["x"], state["scores"], state["expert_scales"], state["table"], state["y"],
                                      state["rows"], fp4=state["fp4"], **state["flags"])
    if op == "ffn":
        # the block updates the residual stream in place: what the attention half leaves there comes first
        hidden = state["hidden"].copy_(state["source"])
        return state["block"].run(0, hidden)
    if state["what"] == "pack":
        if state["storage"] == "fp8":
            return gw.fp8_pack_weights(state["w"], state["scale"])
        packed = gw.nvfp4_pack_weights(state["w"])
        return packed.data, packed.scales, packed.weight_scale
    if state["what"] == "dequantize":
        return gw.nvfp4_dequantize(state["packed"], state["k"], state["n"], output=state["out"])
    return gw.weight_qdq_apply(_lib.QDQ_FP8 if state["storage"] == "fp8" else _lib.QDQ_NVFP4, state["w"])


# --------------------------------------------------------------------------- what it cannot do without

def _touched(rows, skew):
    """Experts that are expected to get a row: every token takes TOPK of EXPERTS, by popularity."""
    popularity = [(i + 1.0) ** -skew for i in range(EXPERTS)]
    total = sum(popularity)
    return sum(1.0 - max(0.0, 1.0 - min(1.0, TOPK * p / total)) ** rows for p in popularity)


def _moe_work(rows, storage, skew):
    per_expert = 3 * INTER * HIDDEN * WEIGHT_BYTES[storage]
    return {"bytes": _touched(rows, skew) * per_expert + rows * (2 * HIDDEN * 2 + EXPERTS * 2),
            "flops": 6.0 * rows * TOPK * HIDDEN * INTER}


def work(case):
    op, storage = case["op"], case["storage"]
    if op == "linear":
        rows, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": n * k * WEIGHT_BYTES[storage] + 2 * rows * (k + n), "flops": 2.0 * rows * k * n}
    if op == "mlp":
        rows, hidden, mlp = case["rows"], case["hidden"], case["mlp"]
        return {"bytes": 3 * hidden * mlp * WEIGHT_BYTES[storage] + 4 * rows * hidden, "flops": 6.0 * rows * hidden * mlp}
    if op == "moe":
        return _moe_work(case["rows"], storage, case["skew"])
    if op == "ffn":
        rows, moe = case["rows"], _moe_work(case["rows"], storage, 0.0)
        # the MoE's input and logits stay inside the block; what comes in and goes out is the residual stream, copied in first
        outer = 2 * rows * HIDDEN * 4 - rows * (2 * HIDDEN * 2 + EXPERTS * 2)
        return {"bytes": moe["bytes"] + outer + 3 * SHARED * HIDDEN * WEIGHT_BYTES[storage] + 2 * EXPERTS * HIDDEN,
                "flops": moe["flops"] + 6.0 * rows * SHARED * HIDDEN + 2.0 * rows * EXPERTS * HIDDEN}
    elements = case["n"] * case["k"]
    if case["what"] == "qdq":
        return {"bytes": 4.0 * elements, "flops": 0.0}
    return {"bytes": elements * (2.0 + WEIGHT_BYTES[storage]), "flops": 0.0}


def tolerance(case):
    """BF16 results of FP32 sums in any order. Between the two projections of an MLP or an expert the activations are
    rounded to FP4 or FP8, where a last-bit difference may become a step; in the feed-forward block, whose router
    logits are BF16, it may also give a token another of two almost equal experts. Weight formats are bit-exact."""
    if case["op"] == "weights":
        return "exact"
    if case["op"] == "linear":
        return {"rel": 5e-3}
    return {"rel": 1e-2, "max": 0.9 if case["op"] == "ffn" else 0.4}
