"""The work this framework is timed on: what a program that serves or trains a model has its
attention do, through the calls such a program makes.

A case is a dict of plain values; `call` says which entry point it goes through:

    "step"     kohaku_tt_b200.decode_step: one token per sequence against a static cache
    "lengths"  kohaku_tt_b200.sdpa with key_lengths, alone or with its gradients
    "dense"    torch.nn.functional.scaled_dot_product_attention, alone or with its gradients
    "packed"   kohaku_tt_b200.sdpa_varlen, alone or with its gradients

Operands are bf16. `listed()` gives the cases that stand for the range, `draw()` more of the
same ranges; FAMILIES below holds both.
"""

import math

import torch
import torch.nn.functional as F

import kohaku_tt_b200 as ktt

# A drawn case does no more work than this (the largest listed case, a packed training step).
MOST_FLOPS = 2.3e12


# ---- the ranges -------------------------------------------------------------------------

def _spread(rng, low, high):
    """A whole number from low to high, spread evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


GROUPED = [(14, 2), (16, 2), (16, 4), (32, 8)]      # query heads, key / value heads
PLAIN = [(8, 8), (12, 12), (16, 16)]


def _draw_decode(rng):
    h, hk = rng.choice(GROUPED + PLAIN)
    return {"call": rng.choice(["step", "lengths"]), "batch": _spread(rng, 1, 64), "heads": h, "kv_heads": hk,
            "dim": rng.choice([64, 128]), "queries": 1, "keys": _spread(rng, 256, 4096), "grad": False, "causal": False}


def _draw_prompt(rng):
    h, hk = rng.choice(GROUPED + PLAIN)
    n = _spread(rng, 32, 4096)
    return {"call": "dense", "batch": _spread(rng, 1, max(1, min(8, 16384 // n))), "heads": h, "kv_heads": hk,
            "dim": rng.choice([64, 128]), "queries": n, "keys": n, "grad": False, "causal": True}


def _draw_image(rng):
    n, h = _spread(rng, 256, 4608), rng.choice([5, 10, 16, 20, 24])
    return {"call": "dense", "batch": rng.choice([1, 2]), "heads": h, "kv_heads": h, "dim": rng.choice([64, 128]),
            "queries": n, "keys": n, "grad": False, "causal": False, "head_views": rng.random() < 0.5}


def _draw_cross(rng):
    h = rng.choice([5, 10, 16, 20])
    return {"call": "dense", "batch": rng.choice([1, 2, 4]), "heads": h, "kv_heads": h, "dim": rng.choice([64, 128]),
            "queries": _spread(rng, 256, 4096), "keys": _spread(rng, 64, 320), "grad": False, "causal": False, "mask": "padding"}


def _draw_masked(rng):
    h, _ = rng.choice(PLAIN)
    n = _spread(rng, 128, 2048)
    return {"call": "dense", "batch": _spread(rng, 1, max(1, min(8, 8192 // n))), "heads": h, "kv_heads": h,
            "dim": rng.choice([64, 128]), "queries": n, "keys": n, "grad": False, "causal": False,
            "mask": rng.choice(["square", "square_bool"])}


def _draw_encoder(rng):
    n, h = _spread(rng, 197, 1536), rng.choice([8, 12, 16])
    return {"call": "dense", "batch": _spread(rng, 1, max(1, min(32, 8192 // n))), "heads": h, "kv_heads": h,
            "dim": rng.choice([80, 96]), "queries": n, "keys": n, "grad": False, "causal": False, "head_views": True}


def _draw_training(rng):
    causal, lengths = rng.random() < 0.6, rng.random() < 0.5
    h, hk = rng.choice(GROUPED + PLAIN)
    n = _spread(rng, 64, 2048)
    return {"call": "lengths" if lengths else "dense", "batch": _spread(rng, 1, max(1, min(16, 8192 // n))), "heads": h,
            "kv_heads": hk, "dim": rng.choice([64, 128]), "queries": n, "keys": n, "grad": True, "causal": causal}


def _draw_packed(rng):
    h, hk = rng.choice([(16, 16), (12, 12), (16, 4)])
    return {"call": "packed", "tokens": _spread(rng, 1024, 65536), "shortest": 64, "longest": _spread(rng, 256, 4096),
            "heads": h, "kv_heads": hk, "dim": rng.choice([64, 128]), "grad": rng.random() < 0.7, "causal": True}


FAMILIES = [
    # Generating text. The smallest call there is: one sequence, one new token, a short cache
    # (what an interactive session pays for every layer of every token) ...
    ([{"name": "generate one", "call": "lengths", "batch": 1, "heads": 14, "kv_heads": 2, "dim": 64, "queries": 1,
       "keys": 1024, "grad": False, "causal": False},
      # ... and a full server batch with the token's neighbours (rotary, cache append), whose
      # time is the reading of the cache.
      {"name": "generate batch", "call": "step", "batch": 64, "heads": 16, "kv_heads": 2, "dim": 128, "queries": 1,
       "keys": 4096, "grad": False, "causal": False}], _draw_decode),
    # Reading a prompt: a short one of an odd length, and the usual benchmark's.
    ([{"name": "prompt short", "call": "dense", "batch": 1, "heads": 14, "kv_heads": 2, "dim": 64, "queries": 77,
       "keys": 77, "grad": False, "causal": True},
      {"name": "prompt", "call": "dense", "batch": 1, "heads": 14, "kv_heads": 2, "dim": 64, "queries": 2048,
       "keys": 2048, "grad": False, "causal": True}], _draw_prompt),
    # Image generation: self-attention of a U-Net level, read in place from its fused
    # projection, and of a transformer over image and text tokens together.
    ([{"name": "image self", "call": "dense", "batch": 2, "heads": 10, "kv_heads": 10, "dim": 64, "queries": 4096,
       "keys": 4096, "grad": False, "causal": False, "head_views": True},
      {"name": "image long", "call": "dense", "batch": 1, "heads": 24, "kv_heads": 24, "dim": 128, "queries": 4396,
       "keys": 4396, "grad": False, "causal": False, "head_views": False}], _draw_image),
    # ... and the cross-attention to the text: few keys, the last of them padding.
    ([{"name": "image cross", "call": "dense", "batch": 2, "heads": 10, "kv_heads": 10, "dim": 64, "queries": 4096,
       "keys": 77, "grad": False, "causal": False, "mask": "padding"}], _draw_cross),
    # A padded batch of prompts whose program hands over a mask with a row per query (causal
    # and padding in one tensor, shared by the heads), as model code written for any backend
    # does.
    ([{"name": "prompt masked", "call": "dense", "batch": 2, "heads": 16, "kv_heads": 16, "dim": 64, "queries": 2048,
       "keys": 2048, "grad": False, "causal": False, "mask": "square"}], _draw_masked),
    # A vision encoder over a batch of pictures: a head dim that is no power of two, a class
    # token that makes the length odd.
    ([{"name": "encoder", "call": "dense", "batch": 16, "heads": 16, "kv_heads": 16, "dim": 80, "queries": 257,
       "keys": 257, "grad": False, "causal": False, "head_views": True}], _draw_encoder),
    # Training, forward and backward: many short sequences, and a right-padded batch with
    # grouped heads.
    ([{"name": "train short", "call": "dense", "batch": 8, "heads": 16, "kv_heads": 16, "dim": 64, "queries": 256,
       "keys": 256, "grad": True, "causal": False},
      {"name": "train padded", "call": "lengths", "batch": 4, "heads": 16, "kv_heads": 4, "dim": 128, "queries": 2048,
       "keys": 2048, "grad": True, "causal": True}], _draw_training),
    # Training on packed sequences: the largest step.
    ([{"name": "train packed", "call": "packed", "tokens": 65536, "shortest": 64, "longest": 4096, "heads": 16,
       "kv_heads": 16, "dim": 128, "grad": True, "causal": True}], _draw_packed),
]


def listed():
    return [dict(case) for cases, _ in FAMILIES for case in cases]


def draw(rng):
    family = rng.choice(FAMILIES)[1]
    while True:
        case = family(rng)
        if _flops(case, _lengths(case, 0)) <= MOST_FLOPS:
            return case


# ---- inputs -----------------------------------------------------------------------------

def _lengths(case, seed):
    """The lengths that a case's sequences have: tokens of each packed sequence, or keys in use
    of each batch row; None where every key is. They are uniform over the range."""
    g = torch.Generator().manual_seed(seed)
    if case["call"] == "packed":
        lengths, left = [], case["tokens"]
        while left > 0:
            n = min(left, int(torch.randint(case["shortest"], case["longest"] + 1, (1,), generator=g)))
            lengths.append(n)
            left -= n
        return lengths
    if case["call"] in ("step", "lengths"):
        # A cache has room for the step's own key.
        high = case["keys"] - 1 if case["call"] == "step" else case["keys"]
        return torch.randint(max(1, case["keys"] // 8), high + 1, (case["batch"],), generator=g).tolist()
    if case.get("mask"):
        return [max(1, case["keys"] - case["keys"] * (b + 1) // (4 * case["batch"])) for b in range(case["batch"])]
    return None


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)


def _heads(g, case, heads, rows):
    """[B, H, S, D] operands: contiguous, or views into a [B, S, H * D] projection."""
    b, d = case["batch"], case["dim"]
    if case.get("head_views"):
        return _normal(g, b, rows, heads * d).view(b, rows, heads, d).transpose(1, 2)
    return _normal(g, b, heads, rows, d)


def _mask(case, lengths):
    """A key-padding mask [B, 1, 1, Sk], or causal and padding together [B, 1, Sq, Sk]: bool
    (True = visible), or added to the logits in the operands' type."""
    keys = torch.arange(case["keys"], device="cuda")
    keep = (keys < torch.tensor(lengths, device="cuda")[:, None])[:, None, None, :]
    if case["mask"] == "padding":
        return keep
    rows = torch.arange(case["queries"], device="cuda")
    keep = keep & (keys <= rows[:, None])
    if case["mask"] == "square_bool":
        return keep
    return torch.zeros(keep.shape, dtype=torch.bfloat16, device="cuda").masked_fill_(~keep, torch.finfo(torch.bfloat16).min)


def prepare(case, seed):
    ktt.install()
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, hk, d = case["heads"], case["kv_heads"], case["dim"]
    lengths = _lengths(case, seed)
    state = {"case": case}
    if case["call"] == "packed":
        n = case["tokens"]
        state["q"], state["k"], state["v"] = _normal(g, n, h, d), _normal(g, n, hk, d), _normal(g, n, hk, d)
        # As a data loader's collation hands them over: offsets on the host.
        state["offsets"] = torch.tensor([0] + lengths, dtype=torch.int32).cumsum(0, dtype=torch.int32)
        if case["grad"]:
            state["dout"] = _normal(g, n, h, d)
    elif case["call"] == "step":
        b, n = case["batch"], case["keys"]
        state["q"], state["k_new"], state["v_new"] = _normal(g, b, h, 1, d), _normal(g, b, hk, 1, d), _normal(g, b, hk, 1, d)
        state["k"], state["v"] = _normal(g, b, hk, n, d), _normal(g, b, hk, n, d)
        state["lengths"] = torch.tensor(lengths, dtype=torch.int32, device="cuda")
        state["next"] = torch.empty_like(state["lengths"])
        turn = torch.arange(n, device="cuda")[:, None] / 10000.0 ** (torch.arange(0, d, 2, device="cuda") / d)
        turn = torch.cat([turn, turn], dim=-1)
        state["cos"], state["sin"] = turn.cos().to(torch.bfloat16), turn.sin().to(torch.bfloat16)
    else:
        state["q"] = _heads(g, case, h, case["queries"])
        state["k"], state["v"] = _heads(g, case, hk, case["keys"]), _heads(g, case, hk, case["keys"])
        if case["grad"]:
            state["dout"] = _heads(g, case, h, case["queries"])
        if case["call"] == "lengths":
            state["lengths"] = torch.tensor(lengths, dtype=torch.int32, device="cuda")
        elif case.get("mask"):
            state["mask"] = _mask(case, lengths)
    if case["grad"]:
        for name in ("q", "k", "v"):
            state[name].requires_grad_(True)
    return state


# ---- one pass ---------------------------------------------------------------------------

def _forward(s):
    case = s["case"]
    if case["call"] == "packed":
        return ktt.sdpa_varlen(s["q"], s["k"], s["v"], s["offsets"], is_causal=case["causal"])
    if case["call"] == "lengths":
        return ktt.sdpa(s["q"], s["k"], s["v"], key_lengths=s["lengths"], is_causal=case["causal"])
    return F.scaled_dot_product_attention(s["q"], s["k"], s["v"], attn_mask=s.get("mask"), is_causal=case["causal"],
                                          enable_gqa=case["heads"] != case["kv_heads"])


def run(s):
    if s["case"]["call"] == "step":
        out = ktt.decode_step(s["q"], s["k_new"], s["v_new"], s["k"], s["v"], s["lengths"], s["cos"], s["sin"], lengths_out=s["next"])
        return {"out": out, "k": s["k"], "v": s["v"], "lengths": s["next"]}
    if s["case"]["grad"]:
        out = _forward(s)
        dq, dk, dv = torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
        return {"out": out, "dq": dq, "dk": dk, "dv": dv}
    with torch.no_grad():
        return _forward(s)


# ---- what a pass cannot do without --------------------------------------------------------

def _triangle(n):
    return n * (n + 1) // 2


def _pairs(case, lengths):
    """Visible (query, key) pairs of one head, over the whole batch."""
    if case["call"] == "packed":
        return sum(_triangle(n) for n in lengths)
    sq, total = case["queries"], 0
    for n in lengths or [case["keys"]] * case["batch"]:
        if case["call"] == "step":
            n += 1
        if case["causal"] or str(case.get("mask", "")).startswith("square"):
            total += _triangle(n) + max(0, sq - n) * n if n <= sq else _triangle(sq)
        else:
            total += sq * n
    return total


def _flops(case, lengths):
    """Two products of 2 D operations per visible pair forward; five of them backward."""
    return (14 if case["grad"] else 4) * case["dim"] * case["heads"] * _pairs(case, lengths)


def work(case):
    lengths = _lengths(case, 0)
    h, hk, d = case["heads"], case["kv_heads"], case["dim"]
    if case["call"] == "packed":
        queries = keys = case["tokens"]
    else:
        queries = case["queries"] * case["batch"]
        keys = sum(lengths) if lengths else case["keys"] * case["batch"]
    rows = queries * h * d * 2
    cells = keys * hk * d * 2
    nbytes = 2 * rows + 2 * cells               # q and out, k and v
    if case["grad"]:
        nbytes += 2 * rows + 2 * cells          # dout and dq, dk and dv
    if case["call"] == "step":
        nbytes += 2 * 2 * case["batch"] * hk * d * 2 + 2 * case["batch"] * d * 2    # the new rows in and out, rotary rows
    if case.get("mask"):
        wide = 2 if case["mask"] == "square" else 1
        nbytes += wide * case["batch"] * case["keys"] * (case["queries"] if case["mask"].startswith("square") else 1)
    return {"bytes": nbytes, "flops": _flops(case, lengths)}


def tolerance(case):
    # bf16 operands and results, fp32 sums; the weights are rounded to bf16 between the two
    # products.
    return {"rel": 1e-2}
