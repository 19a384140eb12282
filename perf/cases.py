"""The work that is timed: what programs built on this package have it do, through its public calls.

``kind`` says which call a case makes:

* ``dense``: ``mmq``, one projection of a batch of tokens by a packed weight;
* ``multi``: ``mmq_multi``, several projections of the same tokens (gate and up of a shared expert);
* ``grouped`` / ``pair``: ``grouped_mmq`` / ``grouped_mmq_pair`` over rows sorted by expert;
* ``moe_mlp``: the feed-forward block over rows sorted by expert (pair, ``silu(gate) * up``, down);
* ``moe_layer``: ``PeerMoEMLP`` on one GPU: routing, the block, the weighted combine;
* ``lm_head``: ``lm_head_loss``, the chunked head with its loss and gradient.

``train`` adds the input gradient, taken by autograd as a training program takes it (for
``moe_layer`` by its ``grad_input``).  Weights are random valid super-blocks whose values have the
spread of trained weights, activations are N(0, 1), expert counts are skewed as a router's are.
"""
import math

import torch

import torch_ggml_ops_b200 as tgo
from torch_ggml_ops_b200.moe_parallel import PeerMoEMLP

Q3_K, Q4_K, Q5_K, Q6_K, IQ2_S = 11, 12, 13, 14, 22
BLOCK_BYTES = {Q3_K: 110, Q4_K: 144, Q5_K: 176, Q6_K: 210, IQ2_S: 82}
FP16_FIELDS = {Q3_K: (108,), Q4_K: (0, 2), Q5_K: (0, 2), Q6_K: (208,), IQ2_S: (0,)}
# super-scale that gives uniformly drawn payload bytes a root mean square of about 0.03
SCALE = {Q3_K: 7e-4, Q4_K: 1e-4, Q5_K: 5e-5, Q6_K: 2.2e-5, IQ2_S: 5e-4}

EXPERTS, HIDDEN, FFN, TOP_K = 256, 2048, 512, 8
VOCAB = 248320
# [out_features, in_features] of the dense projections: attention query, output and narrow (key,
# value, shared gate / up), shared down, and the square and wide ones of the benchmark
DENSE = ((8192, 2048), (2048, 4096), (512, 2048), (2048, 512), (2048, 2048), (4096, 2048))


def listed():
    return [
        # one token of generation through an attention output projection: all latency
        {"name": "decode_1_q4k", "kind": "dense", "qt": Q4_K, "m": 1, "n": 2048, "k": 4096, "train": False},
        # a small decode batch through a shared expert's gate and up
        {"name": "decode_8_gate_up_q5k", "kind": "multi", "qt": Q5_K, "m": 8, "n": 512, "k": 2048, "count": 2, "train": False},
        # logits of a decode batch: every byte of a 417 MB head, few tokens
        {"name": "decode_16_head_q6k", "kind": "dense", "qt": Q6_K, "m": 16, "n": VOCAB, "k": 2048, "train": False},
        # a decode batch through a mixture-of-experts block: some hundred experts of a row or two
        {"name": "decode_16_moe_iq2s_q6k", "kind": "moe_mlp", "qt": IQ2_S, "qt_down": Q6_K, "tokens": 16, "train": False},
        # a short prompt through a square projection
        {"name": "prompt_512_q4k", "kind": "dense", "qt": Q4_K, "m": 512, "n": 2048, "k": 2048, "train": False},
        # a prompt of ragged length through the attention query projection
        {"name": "prompt_1291_q3k", "kind": "dense", "qt": Q3_K, "m": 1291, "n": 8192, "k": 2048, "train": False},
        # a prompt through a mixture-of-experts block: some twenty rows per expert
        {"name": "prompt_600_moe_q3k_q4k", "kind": "moe_mlp", "qt": Q3_K, "qt_down": Q4_K, "tokens": 600, "train": False},
        # fine-tuning, dense projection of a batch of sequences, forward and input gradient
        {"name": "train_4096_iq2s", "kind": "dense", "qt": IQ2_S, "m": 4096, "n": 4096, "k": 2048, "train": True},
        # fine-tuning, one expert projection over the routed rows of 8192 tokens
        {"name": "train_8192_experts_q4k", "kind": "grouped", "qt": Q4_K, "tokens": 8192, "n": FFN, "k": HIDDEN, "train": True},
        # fine-tuning, gate and up of the experts over the routed rows of 16384 tokens
        {"name": "train_16384_pair_q5k", "kind": "pair", "qt": Q5_K, "tokens": 16384, "n": FFN, "k": HIDDEN, "train": True},
        # fine-tuning, loss and gradient of the head, the last chunk ragged
        {"name": "train_600_head_q6k", "kind": "lm_head", "qt": Q6_K, "m": 600, "n": VOCAB, "k": 2048, "train": True},
        # fine-tuning, the whole mixture-of-experts layer from tokens to tokens, 65536 tokens
        {"name": "train_65536_moe_layer", "kind": "moe_layer", "qt": IQ2_S, "qt_down": Q6_K, "tokens": 65536, "train": True},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("dense", "dense", "dense", "dense", "multi", "grouped", "pair", "moe_mlp", "moe_mlp", "moe_layer", "lm_head"))
    qt = rng.choice((Q3_K, Q4_K, Q5_K, Q6_K, IQ2_S))
    down = rng.choice((Q3_K, Q4_K, Q5_K, Q6_K, IQ2_S))
    if kind in ("dense", "multi"):
        n, k = rng.choice(DENSE)
        head = kind == "dense" and rng.random() < 0.2
        if head:
            n, k = _log_int(rng, 32000, VOCAB), 2048
        elif rng.random() < 0.25:   # widths that no tile divides
            n, k = _log_int(rng, 200, 12000), 256 * rng.randint(1, 20)
        m = _log_int(rng, 1, 256 if head else 8192)
        case = {"kind": kind, "qt": qt, "m": m, "n": n, "k": k, "train": m >= 64 and rng.random() < 0.5}
        if kind == "multi":
            case["count"] = rng.randint(2, 4)
        return case
    if kind in ("grouped", "pair"):
        n, k = (HIDDEN, FFN) if kind == "grouped" and rng.random() < 0.5 else (FFN, HIDDEN)
        tokens = _log_int(rng, 1, 16384)
        return {"kind": kind, "qt": qt, "tokens": tokens, "n": n, "k": k, "train": tokens >= 64 and rng.random() < 0.6}
    if kind == "moe_mlp":
        tokens = _log_int(rng, 1, 8192)
        return {"kind": kind, "qt": qt, "qt_down": down, "tokens": tokens, "train": tokens >= 64 and rng.random() < 0.3}
    if kind == "moe_layer":
        tokens = _log_int(rng, 16, 32768)
        return {"kind": kind, "qt": qt, "qt_down": down, "tokens": tokens, "train": tokens >= 64 and rng.random() < 0.6}
    return {"kind": kind, "qt": qt, "m": _log_int(rng, 16, 1024), "n": _log_int(rng, 32000, VOCAB), "k": 2048, "train": True}


# ------------------------------------------------------------------------------ inputs
def _weight(gen, qt, *shape):
    """Packed super-blocks of a weight whose last dimension is ``in_features``."""
    *rows, k = shape
    blocks = torch.randint(0, 256, (math.prod(rows) * (k // 256), BLOCK_BYTES[qt]), dtype=torch.uint8, device="cuda", generator=gen)
    for at in FP16_FIELDS[qt]:
        d = torch.randn(blocks.shape[0], 1, device="cuda", generator=gen).abs_().mul_(SCALE[qt]).half()
        blocks[:, at:at + 2] = d.view(torch.uint8)
    return blocks.reshape(*rows, (k // 256) * BLOCK_BYTES[qt])


def _rows(gen, rows, width, grad=False):
    x = torch.empty(rows, width, dtype=torch.bfloat16, device="cuda").normal_(generator=gen)
    return x.requires_grad_(grad)


def _top_k(gen, tokens):
    """Expert ids [tokens, TOP_K] of a router with favourites."""
    bias = torch.randn(EXPERTS, device="cuda", generator=gen) * 0.5
    return torch.topk(torch.randn(tokens, EXPERTS, device="cuda", generator=gen) * 2.0 + bias, TOP_K).indices


def _groups(gen, tokens):
    """Expert of each group and its end row, every expert a group (some of them empty)."""
    counts = torch.bincount(_top_k(gen, tokens).reshape(-1), minlength=EXPERTS)
    return torch.arange(EXPERTS, device="cuda"), torch.cumsum(counts, 0).to(torch.int32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, qt, train = case["kind"], case["qt"], case["train"]
    s = dict(case)
    if kind in ("dense", "multi"):
        m, n, k, count = case["m"], case["n"], case["k"], case.get("count", 1)
        s["w"] = [_weight(gen, qt, n, k) for _ in range(count)]
        s["x"] = _rows(gen, m, k, train)
        s["dy"] = [_rows(gen, m, n) for _ in range(count)] if train else None
    elif kind in ("grouped", "pair"):
        n, k, count = case["n"], case["k"], 2 if kind == "pair" else 1
        s["w"] = [_weight(gen, qt, EXPERTS, n, k) for _ in range(count)]
        s["ids"], s["ends"] = _groups(gen, case["tokens"])
        s["x"] = _rows(gen, case["tokens"] * TOP_K, k, train)
        s["dy"] = [_rows(gen, case["tokens"] * TOP_K, n) for _ in range(count)] if train else None
    elif kind in ("moe_mlp", "moe_layer"):
        tokens = case["tokens"]
        w = [_weight(gen, qt, EXPERTS, FFN, HIDDEN), _weight(gen, qt, EXPERTS, FFN, HIDDEN),
             _weight(gen, case["qt_down"], EXPERTS, HIDDEN, FFN)]
        if kind == "moe_mlp":
            s["w"] = w
            s["ids"], s["ends"] = _groups(gen, tokens)
            s["x"] = _rows(gen, tokens * TOP_K, HIDDEN, train)
            s["dy"] = _rows(gen, tokens * TOP_K, HIDDEN) if train else None
        else:
            s["layer"] = PeerMoEMLP(*w, qt, case["qt_down"], EXPERTS, HIDDEN, FFN, capacity_rows=tokens * TOP_K,
                                    tokens_per_rank=tokens, top_k=TOP_K)
            s["top_k"] = _top_k(gen, tokens).to(torch.int32)
            gate = torch.rand(tokens, TOP_K, device="cuda", generator=gen) + 0.25
            s["gate"] = gate / gate.sum(1, keepdim=True)
            s["x"] = _rows(gen, tokens, HIDDEN)
            s["dy"] = _rows(gen, tokens, HIDDEN) if train else None
    else:
        s["w"] = _weight(gen, qt, case["n"], case["k"])
        s["x"] = _rows(gen, case["m"], case["k"])
        s["targets"] = torch.randint(0, case["n"], (case["m"],), device="cuda", generator=gen)
    return s


# ------------------------------------------------------------------------------ one pass
def run(state):
    s = state
    kind, qt, x = s["kind"], s["qt"], s["x"]
    if kind == "lm_head":
        return tgo.lm_head_loss(x, s["w"], qt, s["n"], s["targets"])
    if kind == "moe_layer":
        layer = s["layer"]
        layer.plan(s["top_k"], s["gate"])
        y = layer.forward(x)
        return (y, layer.grad_input(s["dy"])) if s["train"] else y
    if kind == "dense":
        y = (tgo.mmq(x, s["w"][0], qt, s["n"]),)
    elif kind == "multi":
        y = tgo.mmq_multi(x, s["w"], qt, s["n"])
    elif kind == "grouped":
        y = (tgo.grouped_mmq(x, s["w"][0], s["ids"], s["ends"], qt, s["n"]),)
    elif kind == "pair":
        y = tgo.grouped_mmq_pair(x, *s["w"], s["ids"], s["ends"], qt, s["n"])
    else:
        y = (tgo.moe_mlp(x, *s["w"], s["ids"], s["ends"], qt, s["qt_down"], FFN),)
    if not s["train"]:
        return y
    dy = s["dy"] if isinstance(s["dy"], list) else [s["dy"]]
    return *[t.detach() for t in y], *torch.autograd.grad(y, x, dy)


# ------------------------------------------------------------------------------ what a pass needs
def _packed(qt, n, k):
    return n * (k // 256) * BLOCK_BYTES[qt]


def work(case):
    """Every input once, every output once; the multiplications of the directions that are run.
    Weights: those of the experts that the tokens are expected to hit."""
    kind, qt, train = case["kind"], case["qt"], case["train"]
    ways = 2 if train else 1
    if kind in ("dense", "multi", "lm_head"):
        m, n, k, count = case["m"], case["n"], case["k"], case.get("count", 1)
        weight, flops = count * _packed(qt, n, k), 2.0 * m * n * k * count
        if kind == "lm_head":   # the logits need not leave the chip
            return {"bytes": weight + m * k * 4 + m * 8 + 4, "flops": ways * flops}
        return {"bytes": weight + ways * 2 * m * (k + count * n), "flops": ways * flops}
    tokens = case["tokens"]
    rows = tokens * TOP_K
    hit = EXPERTS * (1.0 - (1.0 - TOP_K / EXPERTS) ** tokens)
    if kind in ("grouped", "pair"):
        n, k, count = case["n"], case["k"], 2 if kind == "pair" else 1
        return {"bytes": hit * count * _packed(qt, n, k) + ways * 2 * rows * (k + count * n) + EXPERTS * 12,
                "flops": ways * 2.0 * rows * n * k * count}
    weight = hit * (2 * _packed(qt, FFN, HIDDEN) + _packed(case["qt_down"], HIDDEN, FFN))
    flops = ways * 6.0 * rows * FFN * HIDDEN
    if kind == "moe_mlp":
        return {"bytes": weight + ways * 4 * rows * HIDDEN + EXPERTS * 12, "flops": flops}
    return {"bytes": weight + ways * 4 * tokens * HIDDEN + rows * 8, "flops": flops}


def tolerance(case):
    """bf16 results: one rounding (2^-9 of a value) and, for another order of the fp32 sums, now and
    then the neighbouring value.  Chains round between their matmuls too, and the head's gradient
    goes through exponentials of bf16 logits."""
    if case["kind"] in ("dense", "grouped", "pair"):
        return {"rel": 4e-3, "max": 0.02}
    if case["kind"] == "multi":   # gradients of several weights are added in bf16
        return {"rel": 6e-3, "max": 0.05}
    return {"rel": 1e-2, "max": 0.1}
