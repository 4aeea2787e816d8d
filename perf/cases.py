"""The work a user of this library has it do, as cases that can be timed and compared.

A case is one pass of an expert layer (or of the weight packer) through the public entry
points, called as a serving program calls them: buffers, locks and packed weights are
kept between passes, routing and activations are new on every pass, nothing synchronises.
Weights are INT4 with BF16 scales per 32 input channels, drawn in checkpoint form
(uniform codes, scales uniform in [0.005, 0.02]); activations are BF16 N(0, 1).

``hidden`` / ``inter`` are the layer's widths: the gate_up weight is
[experts, 2 * inter, hidden], the down weight [experts, hidden, inter].  ``experts`` of
``experts_total`` are held locally; the router spreads every token over ``top_k`` of
``experts_total`` and only local routes are computed.

Kinds:
  steps       moe_align_block_size -> indexed (gate_up) -> silu_mul -> indexed (down)
  fused       moe_align_block_size -> indexed_gate_up_silu -> indexed (down)
  contiguous  contiguous (gate_up) -> silu_mul -> contiguous (down)
  masked      masked (gate_up) -> silu_mul -> masked (down)
  pack        pack_w4a16 of one weight
"""

import math

import torch

import chord_b200
from chord_b200 import fused_ops, indexed_gemm

# Layer widths of the benchmark's model (48 of 384 experts per GPU under EP8, 24 under
# EP16, 12 under EP32), top_k 8.
HIDDEN, INTER, TOP_K, TOTAL = 7168, 2048, 8, 384


def listed():
    ep8 = dict(experts=48, experts_total=TOTAL, hidden=HIDDEN, inter=INTER, top_k=TOP_K)
    ep16 = dict(experts=24, experts_total=TOTAL, hidden=HIDDEN, inter=INTER)
    return [
        # A small layer (8 experts, 512 wide): nothing but launch and call latency.
        dict(name="small_layer", kind="steps", experts=8, experts_total=8, hidden=512, inter=512, top_k=2,
             tokens=64),
        # Decode under EP8 at the benchmark's four batch sizes: 1 (one interactive user; one
        # or two local experts reached), 16, 64 and 256 tokens (every local expert reached).
        dict(name="decode_1", kind="steps", tokens=1, **ep8),
        dict(name="decode_16", kind="steps", tokens=16, **ep8),
        dict(name="decode_64", kind="steps", tokens=64, **ep8),
        dict(name="decode_256", kind="steps", tokens=256, **ep8),
        # Decode with every route local (the rows an EP rank sees after dispatch), an odd
        # count, SiLU*mul fused into gate_up.
        dict(name="decode_local_37", kind="fused", tokens=37, **{**ep8, "experts_total": 48}),
        # Prefill of one sequence of 4096 tokens through the routed entry points (about 85
        # rows for each local expert).
        dict(name="prefill_4096", kind="fused", tokens=4096, **ep8),
        # Prefill in the grouped layout: 8192 tokens with uneven expert popularity (many
        # experts with fewer rows than a block, a few with a thousand), and a large even one
        # (the largest case).
        dict(name="contiguous_uneven", kind="contiguous", tokens=8192, popularity=0.5, **ep8),
        dict(name="contiguous_even", kind="contiguous", tokens=24000, popularity=0.0, **ep8),
        # Decode in the masked layout at EP16: fixed [24, 256, hidden] buffers, a few rows or
        # about half of them filled.
        dict(name="masked_8", kind="masked", expected_m=8, max_m=256, **ep16),
        dict(name="masked_128", kind="masked", expected_m=128, max_m=256, **ep16),
        # Loading a checkpoint: one weight of sixteen experts, eight codes per word.
        dict(name="pack_checkpoint", kind="pack", experts=16, n=2 * INTER, k=HIDDEN, packed=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case: half of them decode, the rest spread over the other kinds; half with
    the benchmark's layer, half with other widths, expert counts and top_k."""
    kind = rng.choice(["steps", "steps", "steps", "fused", "fused", "contiguous", "masked", "masked", "pack"])
    if rng.random() < 0.5:
        layer = dict(experts=rng.choice([12, 24, 48]), experts_total=TOTAL, hidden=HIDDEN, inter=INTER)
        top_k = TOP_K
    else:
        # gate_up fused with SiLU*mul needs whole 128-row blocks of gate rows
        unit = 128 if kind == "fused" else 64
        experts = rng.randint(4, 64)
        layer = dict(experts=experts, experts_total=experts * rng.choice([1, 1, 2, 8]),
                     hidden=128 * rng.randint(8, 48), inter=unit * rng.randint(512 // unit, 2048 // unit))
        top_k = rng.randint(1, 8) if layer["experts_total"] >= 8 else rng.randint(1, 4)
    if kind == "pack":
        return dict(kind=kind, experts=rng.randint(1, 16), n=128 * rng.randint(2, 32),
                    k=64 * rng.randint(4, 112), packed=rng.random() < 0.7)
    if kind == "masked":
        expected = _log_int(rng, 1, 200)
        return dict(kind=kind, expected_m=expected, max_m=rng.choice([256, 384]), **layer)
    if kind == "contiguous":
        tokens = _log_int(rng, 256, 16384)
        popularity = rng.choice([0.0, 0.5, 2.0])
    else:
        tokens = _log_int(rng, 1, 512) if rng.random() < 0.75 else _log_int(rng, 512, 8192)
        popularity = None
    # at most 24000 local rows, the largest listed case's
    rows = tokens * top_k * layer["experts"] / layer["experts_total"]
    if rows > 20000:
        tokens = max(1, int(tokens * 20000 / rows))
    case = dict(kind=kind, tokens=tokens, top_k=top_k, **layer)
    if popularity is not None:
        case["popularity"] = popularity
    return case


# --------------------------------------------------------------------- inputs --

def _checkpoint(experts, n, k, g):
    words = torch.randint(-2**31, 2**31 - 1, (experts, n, k // 8), dtype=torch.int32, device="cuda", generator=g)
    scale = torch.rand((experts, n, k // 32), device="cuda", generator=g).mul_(0.015).add_(0.005)
    return words, scale.to(torch.bfloat16)


def _weight(experts, n, k, g):
    return chord_b200.pack_w4a16(*_checkpoint(experts, n, k, g), packed=True)


def _normal(shape, g):
    return torch.randn(shape, device="cuda", generator=g, dtype=torch.bfloat16)


def _popularity(case, experts, g):
    """Even, or drawn from Dirichlet(popularity) (up to its norm)."""
    alpha = case.get("popularity", 0.0)
    if alpha == 0:
        return torch.ones(experts, device="cuda")
    return torch._standard_gamma(torch.full((experts,), float(alpha), device="cuda"), generator=g).clamp_(min=1e-12)


def _topk(case, g, base):
    """int32 [tokens, top_k]: distinct experts per token, uniform over all experts.  The first
    token reaches a local expert."""
    scores = torch.randn((case["tokens"], case["experts_total"]), device="cuda", generator=g)
    first = int(torch.randint(case["experts"], (1,), device="cuda", generator=g))
    scores[0, base + first] += 1e6
    return scores.topk(case["top_k"], dim=1).indices.to(torch.int32).contiguous()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "pack":
        words, scale = _checkpoint(case["experts"], case["n"], case["k"], g)
        if not case["packed"]:
            shifts = torch.arange(0, 32, 4, dtype=torch.int32, device="cuda")
            words = ((words.unsqueeze(-1) >> shifts) & 15).view(case["experts"], case["n"], case["k"])
        state.update(words=words, scale=scale, packed=case["packed"])
        return state
    experts, hidden, inter = case["experts"], case["hidden"], case["inter"]
    state["w13"] = _weight(experts, 2 * inter, hidden, g)
    state["w2"] = _weight(experts, hidden, inter, g)

    def buffers(rows, *widths):
        # rows that no route names stay as they are: zero
        return [torch.zeros((rows, w), dtype=torch.bfloat16, device="cuda") for w in widths]

    if kind == "masked":
        max_m = case["max_m"]
        counts = torch.poisson(torch.full((experts,), float(case["expected_m"]), device="cuda"), generator=g)
        counts[0].clamp_(min=1)
        state["masked_m"] = counts.clamp_(max=max_m).to(torch.int32)
        state["expected_m"] = case["expected_m"]
        state["x"] = _normal((experts, max_m, hidden), g)
        state["gate_up"], state["act"], state["out"] = buffers(experts * max_m, 2 * inter, inter, hidden)
        return state
    base = (case["experts_total"] // case["experts"] // 2) * experts  # a rank in the middle
    if kind == "contiguous":
        # as many local rows as the router sends on average, over experts of even or uneven
        # popularity; the buffer holds them with every expert's run padded to 128 rows
        rows = max(1, case["tokens"] * case["top_k"] * experts // case["experts_total"])
        popularity = _popularity(case, experts, g)
        owner = torch.multinomial(popularity, rows, replacement=True, generator=g)
        index = []
        for e, c in enumerate(torch.bincount(owner, minlength=experts).tolist()):
            index += [e] * c + [-1] * (-c % 128)
        index += [-1] * ((rows // 128 + experts) * 128 - len(index))
        state["m_indices"] = torch.tensor(index, dtype=torch.int32, device="cuda")
        state["x"] = _normal((len(index), hidden), g)
        state["x"][state["m_indices"] < 0] = 0
        state["gate_up"], state["act"], state["out"] = buffers(len(index), 2 * inter, inter, hidden)
        return state
    state.update(topk_ids=_topk(case, g, base), tokens=case["tokens"], top_k=case["top_k"], experts=experts,
                 base=base, total=case["experts_total"], x=_normal((case["tokens"], hidden), g),
                 locks=torch.zeros(1024, dtype=torch.int32, device="cuda"))
    rows = case["tokens"] * case["top_k"]
    state["gate_up"], state["act"], state["out"] = buffers(rows, 2 * inter if kind == "steps" else 0, inter, hidden)
    return state


# ----------------------------------------------------------------------- pass --

def run(state):
    kind = state["kind"]
    if kind == "pack":
        weight = chord_b200.pack_w4a16(state["words"], state["scale"], packed=state["packed"])
        return weight.packed, weight.scale
    w13, w2 = state["w13"], state["w2"]
    gate_up, act, out = state["gate_up"], state["act"], state["out"]
    if kind == "masked":
        masked_m, expected_m = state["masked_m"], state["expected_m"]
        chord_b200.masked(state["x"], w13, masked_m, expected_m, outputs=gate_up)
        fused_ops.silu_mul(gate_up, outputs=act)
        chord_b200.masked(act, w2, masked_m, expected_m, outputs=out)
        return gate_up, out
    if kind == "contiguous":
        m_indices = state["m_indices"]
        chord_b200.contiguous(state["x"], w13, m_indices, outputs=gate_up)
        fused_ops.silu_mul(gate_up, outputs=act)
        chord_b200.contiguous(act, w2, m_indices, outputs=out)
        return gate_up, out
    top_k, locks = state["top_k"], state["locks"]
    block_m = chord_b200.indexed_block_m(w13, state["tokens"], top_k, total_experts=state["total"])
    routing = fused_ops.moe_align_block_size(state["topk_ids"], block_m, state["experts"],
                                             expert_base=state["base"])
    if kind == "steps":
        chord_b200.indexed(state["x"], w13, *routing, top_k, locks=locks, outputs=gate_up, block_m=block_m)
        fused_ops.silu_mul(gate_up, sorted_ids=routing[0], num_tokens_padded=routing[2], outputs=act)
    else:
        indexed_gemm.indexed_gate_up_silu(state["x"], w13, *routing, top_k, locks=locks, outputs=act,
                                          block_m=block_m)
    chord_b200.indexed(act, w2, *routing, 1, locks=locks, outputs=out, block_m=block_m)
    return (gate_up, out) if kind == "steps" else (act, out)


# ----------------------------------------------------------------------- cost --

def _local_rows_and_experts(case):
    """Expected local rows and expected number of local experts that get one."""
    experts = case["experts"]
    if case["kind"] == "masked":
        return experts * min(case["expected_m"], case["max_m"]), experts * (1 - math.exp(-case["expected_m"]))
    total, top_k = case["experts_total"], case["top_k"]
    rows = max(1.0, case["tokens"] * top_k * experts / total)
    reached = max(1.0, experts * (1 - (1 - top_k / total) ** case["tokens"])) if top_k < total else experts
    return rows, reached


def work(case):
    """Every reached expert's weights and scales, activation rows in, result rows out (the
    intermediate between the two projections in and out once each where they are separate
    calls), and the multiplications of the routed rows."""
    if case["kind"] == "pack":
        codes = case["experts"] * case["n"] * case["k"]
        scales = codes // 32 * 2
        return {"bytes": codes * (0.5 if case["packed"] else 4) + codes * 0.5 + 2 * scales, "flops": 0}
    rows, reached = _local_rows_and_experts(case)
    hidden, inter = case["hidden"], case["inter"]
    weights = reached * 3 * inter * hidden * (0.5 + 2 / 32)
    read = rows if case["kind"] in ("masked", "contiguous") else min(rows, case["tokens"])
    moved = 2 * (read * hidden + rows * hidden + 2 * rows * inter)
    if case["kind"] != "fused":
        moved += 2 * rows * 2 * inter * 2  # gate_up written and read back
    return {"bytes": weights + moved, "flops": 2 * rows * 3 * inter * hidden}


def tolerance(case):
    if case["kind"] == "pack":
        return "exact"
    # BF16 results of FP32 sums over BF16 products.  The same layer in FP64, with unrounded
    # (code - 8) * scale weights and an unrounded intermediate, differs from the library's
    # by rel 2.2e-3 after gate_up and 4.4e-3 after down, max 0.018-0.076 (the largest of
    # some ten million values); with the weights and the intermediate rounded to BF16 by
    # rel 1.7e-3, max 0.013.
    return {"rel": 1.6e-2, "max": 0.3}
