"""Workloads of the library on one GPU, as a program that uses it runs them.

Four kinds of call, each through the public entry points:

* ``train``  one MoE layer, forward and backward, through ``stream_moe_func`` and autograd
* ``infer``  the forward alone, under ``torch.no_grad``
* ``comm``   the stand-alone exchange of a custom expert layer: ``Buffer.dispatch``, ``combine`` and, with
             ``grads``, ``dispatch_grads`` and ``combine_grads``
* ``route``  ``router_topk``: linear gate, softmax, top-k, rank bitmap

Routing is an input of the layer and exchange cases (it is computed by the router, which has cases of its own), so a
near-tie of two gate logits cannot decide what is compared.  Everything is bf16 with fp32 top-k weights: the library
takes no other type.
"""
import math

import torch

from streamep_b200.models.moe_layer import make_buffer
from streamep_b200.ops.grouped_gemm import compress_pool_to_recv, router_topk
from streamep_b200.stream_moe import make_streams, stream_moe_func

#: Upper ends of the ranges that ``draw`` samples.
MAX_TOKENS, MAX_HIDDEN, MAX_EXPERTS, MAX_TOPK = 16384, 7168, 64, 8


def listed():
    return [
        # The benchmark's default layer: a long training sequence, fixed receive regions (no host read of the sizes).
        dict(name="train default layer", kind="train", tokens=8192, hidden=2048, ffn=1408, experts=8, topk=6, level=0,
             capacity=True, routing="gate", skip=0.0),
        # The benchmark's Mixtral-style sweep shape, one of its layers: few, very wide experts, the largest call.
        dict(name="train wide experts", kind="train", tokens=16384, hidden=4096, ffn=14336, experts=8, topk=2, level=0,
             capacity=False, routing="gate", skip=0.0),
        # The benchmark's stress shape on one rank: an odd token count, hot experts, the forward GEMM recomputed.
        dict(name="train skewed recompute", kind="train", tokens=5003, hidden=7168, ffn=2048, experts=32, topk=8, level=1,
             capacity=False, routing="zipf", skip=0.0),
        # Many small experts (the shape of the reference's production comments, one rank's share), a short batch.
        dict(name="train many small experts", kind="train", tokens=2048, hidden=3072, ffn=768, experts=32, topk=8, level=0,
             capacity=True, routing="gate", skip=0.0),
        # Ragged sizes: nothing is a multiple of a tile, some pairs are skipped (-1), the pool is rebuilt in backward.
        dict(name="train ragged", kind="train", tokens=1777, hidden=1000, ffn=520, experts=12, topk=3, level=2,
             capacity=False, routing="gate", skip=0.05),
        # The benchmark's tiny layer: unit tests, debugging runs and small models; launches and host time.
        dict(name="train tiny", kind="train", tokens=512, hidden=256, ffn=128, experts=4, topk=2, level=0,
             capacity=False, routing="gate", skip=0.0),
        # Decoding a small batch: the smallest layer call, bound by reading the weights and by latency.
        dict(name="infer decode", kind="infer", tokens=16, hidden=2048, ffn=1408, experts=8, topk=6, level=0,
             capacity=True, routing="gate", skip=0.0),
        # Decoding a larger batch on the benchmark's dispatch-heavy shape: a few rows for each of 32 experts.
        dict(name="infer decode wide", kind="infer", tokens=96, hidden=7168, ffn=2048, experts=32, topk=8, level=0,
             capacity=True, routing="gate", skip=0.0),
        # Prefill / evaluation of a sequence of odd length, exactly sized buffers.
        dict(name="infer prefill", kind="infer", tokens=4001, hidden=3072, ffn=768, experts=32, topk=8, level=0,
             capacity=False, routing="gate", skip=0.0),
        # The communication benchmark's shape: all four stand-alone exchanges.
        dict(name="comm round trip", kind="comm", tokens=4096, hidden=7168, ffn=0, experts=32, topk=8, grads=True,
             routing="uniform", skip=0.0),
        # The router in front of the default layer on eight ranks' worth of experts.
        dict(name="route sequence", kind="route", tokens=8192, hidden=2048, experts=64, topk=6, ranks=8, probs=False),
        # The router of a decoding step with many experts.
        dict(name="route decode", kind="route", tokens=64, hidden=7168, experts=256, topk=8, ranks=8, probs=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A row width: mostly a multiple of 64 as models have them, sometimes only of 8 (what the library asks for)."""
    step = 64 if rng.random() < 0.75 else 8
    return max(lo, min(hi, _log_int(rng, lo, hi) // step * step))


def _draw_once(rng):
    kind = rng.choices(["train", "infer", "comm", "route"], [9, 6, 2, 3])[0]
    if kind == "route":
        experts = rng.choice([8, 16, 32, 64, 128, 256, rng.randrange(1, 33) * 8])
        return dict(kind=kind, tokens=_log_int(rng, 1, MAX_TOKENS), hidden=_width(rng, 256, MAX_HIDDEN), experts=experts,
                    topk=rng.randint(1, min(MAX_TOPK, experts)), ranks=rng.choice([1, 2, 4, 8]), probs=rng.random() < 0.2)
    experts = rng.choice([4, 8, 8, 16, 32, 64, rng.randint(2, MAX_EXPERTS)])
    case = dict(kind=kind, tokens=_log_int(rng, 1 if kind == "infer" else 64, MAX_TOKENS), hidden=_width(rng, 256, MAX_HIDDEN),
                ffn=0 if kind == "comm" else _width(rng, 128, 14336), experts=experts,
                topk=rng.randint(1, min(MAX_TOPK, experts)), routing=rng.choice(["gate", "gate", "uniform", "zipf"]),
                skip=rng.choice([0.0, 0.0, 0.05]))
    if kind == "comm":
        case["grads"], case["skip"] = rng.random() < 0.7, 0.0
    else:
        case["capacity"] = rng.random() < 0.6
        case["level"] = rng.choice([0, 0, 0, 1, 2]) if kind == "train" else 0
    return case


def draw(rng):
    """One more case of the same ranges, never more work than the largest listed one of its kind."""
    limit = {}
    for c in listed():
        w = work(c)
        have = limit.get(c["kind"], (0, 0))
        limit[c["kind"]] = (max(have[0], w["bytes"]), max(have[1], w["flops"]))
    while True:
        case = _draw_once(rng)
        w, (most_bytes, most_flops) = work(case), limit[case["kind"]]
        if w["bytes"] <= most_bytes and w["flops"] <= most_flops:
            return case


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _normal(gen, shape, std):
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=gen)


def _routing(gen, case, x):
    """Distinct experts per token and their weights: from a linear gate on x, uniform, or Zipf(1.2) over expert ids."""
    T, E, K = case["tokens"], case["experts"], case["topk"]
    if case["routing"] == "gate":
        gate = torch.randn(E, case["hidden"], generator=gen, device="cuda") * 0.02
        score = x.float() @ gate.t()
        weights, idx = score.topk(K, dim=1)
        weights = torch.softmax(weights, dim=1)
    else:
        score = -torch.log(-torch.log(torch.rand(T, E, generator=gen, device="cuda").clamp_(1e-9, 1 - 1e-7)))
        if case["routing"] == "zipf":
            score = score - 1.2 * torch.log(torch.arange(1, E + 1, device="cuda", dtype=torch.float32))
        idx = score.topk(K, dim=1).indices
        weights = torch.softmax(torch.randn(T, K, generator=gen, device="cuda"), dim=1)
    if case["skip"] > 0:
        idx = torch.where(torch.rand(T, K, generator=gen, device="cuda") < case["skip"], torch.full_like(idx, -1), idx)
    return idx.contiguous(), weights.contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    T, H, E, K = case["tokens"], case["hidden"], case["experts"], case["topk"]
    s = {"case": dict(case), "x": _normal(gen, (T, H), 1.0)}
    if case["kind"] == "route":
        s["gate"] = _normal(gen, (E, H), 0.02)
        s["buffer"] = make_buffer(None, T, 256, 1, 8)      # a program's router reports into its layer's buffer
        return s
    s["idx"], s["weights"] = _routing(gen, case, s["x"])
    s["buffer"] = make_buffer(None, T, H, K, E, capacity_factor=1.5 if case.get("capacity") else None)
    if case["kind"] == "comm":
        s["rows"] = s["buffer"].alloc_symmetric([int((s["idx"] >= 0).any(dim=1).sum()), H], torch.bfloat16)
        s["rows"].normal_(0.0, 1.0, generator=gen)
        if case["grads"]:
            tiles = sum((n + 127) // 128 for n in torch.bincount(s["idx"][s["idx"] >= 0], minlength=E).tolist())
            s["dy"] = _normal(gen, (T, H), 0.1)
            s["slot_grads"] = torch.randn(tiles * 128, generator=gen, device="cuda")
            s["done"] = torch.ones(s["rows"].shape[0], dtype=torch.int64, device="cuda")
        return s
    s["streams"] = make_streams()
    s["w1"] = _normal(gen, (E, 2 * case["ffn"], H), 0.02)
    s["w2"] = _normal(gen, (E, H, case["ffn"]), 0.02)
    if case["kind"] == "train":
        s["dy"] = _normal(gen, (T, H), 0.1)
        for name in ("x", "weights", "w1", "w2"):
            s[name].requires_grad_(True)
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def _layer(s):
    c = s["case"]
    return stream_moe_func(s["buffer"], s["x"], s["idx"], s["weights"], None, s["w1"], s["w2"], streams=s["streams"],
                           num_experts=c["experts"], activation_checkpoint_level=c["level"])


def run(s):
    c, buf = s["case"], s["buffer"]
    if c["kind"] == "train":
        out = _layer(s)
        grads = torch.autograd.grad(out, (s["x"], s["weights"], s["w1"], s["w2"]), s["dy"])
        return (out.detach(),) + grads
    if c["kind"] == "infer":
        with torch.no_grad():
            return _layer(s)
    if c["kind"] == "route":
        return router_topk(s["x"], s["gate"], c["topk"], num_ranks=c["ranks"], return_probs=c["probs"], buffer=buf)
    # What the pools hold is returned as one row per received token (padding rows of a pool are not written).  The
    # program's own expert kernels would stamp the finished tokens; here all of them are finished.
    pool, h, _ = buf.dispatch(s["x"], s["idx"], s["weights"], None, c["experts"])
    got = {"rows": compress_pool_to_recv(pool, h.pool_recv_token, h.num_recv_tokens, buffer=buf),
           "slots": h.recv_token_to_slots, "weights": h.pool_topk_weight[h.recv_token_to_slots], "frequency": h.expert_frequency}
    h.y_done_per_token.fill_(1)
    got["out"], _ = buf.combine(s["rows"], h, combine_seq=1)
    if c["grads"]:
        grad_pool, _, _ = buf.dispatch_grads(h, s["dy"])
        got["grad_rows"] = compress_pool_to_recv(grad_pool, h.pool_recv_token, h.num_recv_tokens, buffer=buf)
        got["dx"], got["dweights"] = buf.combine_grads(s["rows"], h, s["slot_grads"], s["done"], dispatch_seq=1)
    return got


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how close two correct passes are
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    T, H, E, K = case["tokens"], case["hidden"], case["experts"], case["topk"]
    pairs = T * K * (1.0 - case.get("skip", 0.0))
    token_rows, pair_rows = 2.0 * T * H, 2.0 * pairs * H
    routing = 12.0 * T * K
    if case["kind"] == "route":
        outs = routing + T * case["ranks"] + (4.0 * T * E if case["probs"] else 0.0)
        return {"bytes": token_rows + 2.0 * E * H + outs, "flops": 2.0 * T * H * E}
    if case["kind"] == "comm":
        # each direction: rows in, one row per pair out, one row per token back in, reduced rows out, and the rows
        # read back out of the pool
        ways = 2.0 if case["grads"] else 1.0
        return {"bytes": ways * (pair_rows + 5.0 * token_rows) + routing, "flops": 0.0}
    weights = 2.0 * 3.0 * H * case["ffn"] * min(E, max(pairs, 1.0))    # only the experts that some pair can reach
    if case["kind"] == "infer":
        return {"bytes": weights + 2.0 * token_rows + routing, "flops": 6.0 * pairs * H * case["ffn"]}
    recompute = 4.0 if case["level"] > 0 else 0.0
    return {"bytes": 2.0 * 2.0 * 3.0 * H * case["ffn"] * E + 4.0 * token_rows + 2.0 * routing,
            "flops": (18.0 + recompute) * pairs * H * case["ffn"]}


def tolerance(case):
    if case["kind"] == "comm":
        return "exact"                       # rows are moved, not computed: one bf16 row (and one scalar) per source
    if case["kind"] == "route":
        # fp32 sums over hidden <= 7168 exact products, then a softmax; logits nearer than their rounding may swap
        return {"rel": 2e-5, "max": 1e-3, "differ": 1e-3}
    return {"rel": 1e-2}                     # bf16 rows, weights and gradients, fp32 accumulation
