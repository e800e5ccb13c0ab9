"""The calls that are timed: the quantized linear layers of a decoder, as a program that serves one makes them.

Five kinds of work, each through the public functions of ``ignis_b200``:

``nvfp4_linear``   one ``nvfp4.linear`` over an [n, k] parent
``nvfp4_layer``    the linear work of one dense decoder layer with hidden 5120 in NVFP4: the q | k | v
                   parent, the output projection and the MLP added to the residual stream
``trellis_linear`` one ``trellis.linear`` (the output head among them)
``trellis_layer``  the same dense layer in the trellis format
``moe_block``      one mixture-of-experts block: router, routed experts, shared expert, combine

Tokens run from 1 (one sequence decoding) over some dozens (batched decode, verification of drafts, the
rest of a prompt) to 4096 or 8192 (a prompt chunk). Weights have the distributions of the repository's
benchmark: NVFP4 codes uniform over the 16 values with scales E4M3(|N(0,1)| + 0.1), trellis words
uniform, activations N(0,1) in BF16, expert popularity Zipf(1.1).
"""
from __future__ import annotations

import math

import torch

from ignis_b200 import moe, nvfp4, trellis

# the dense layer: (out, in) of each projection
HIDDEN, Q, KV, INTER = 5120, 6144, 1024, 17408
QKV_ROWS = [Q, KV, KV]
HEAD = 248320                                           # the output head's width
LAYER_SHAPES = [(Q, HIDDEN), (KV, HIDDEN), (Q + 2 * KV, HIDDEN), (HIDDEN, Q), (INTER, HIDDEN), (2 * INTER, HIDDEN), (HIDDEN, INTER)]
DENSE_PARAMS = sum(QKV_ROWS) * HIDDEN + HIDDEN * Q + 3 * INTER * HIDDEN
# (hidden, intermediate, experts, choices per token) of the two expert geometries in use
MOE_GEOMETRIES = [(2048, 768, 512, 10), (2560, 640, 512, 10)]
ZIPF = 1.1
POLICIES = {"a16": nvfp4.A16_ONLY, "a4": nvfp4.ALLOW_A4}


def listed() -> list[dict]:
    return [
        # the smallest call: a key projection for one decoding sequence; the call itself costs most
        {"name": "nvfp4_kv_t1", "kind": "nvfp4_linear", "n": KV, "k": HIDDEN, "tokens": 1, "policy": "a16"},
        # one sequence decoding, activations kept in BF16
        {"name": "nvfp4_layer_t1_a16", "kind": "nvfp4_layer", "tokens": 1, "policy": "a16"},
        # eight sequences decoding, under both activation policies
        {"name": "nvfp4_layer_t8_a16", "kind": "nvfp4_layer", "tokens": 8, "policy": "a16"},
        {"name": "nvfp4_layer_t8_a4", "kind": "nvfp4_layer", "tokens": 8, "policy": "a4"},
        # a short prompt, or many sequences verifying drafts: an odd width between decode and prefill
        {"name": "nvfp4_layer_t77_a4", "kind": "nvfp4_layer", "tokens": 77, "policy": "a4"},
        # the ragged last chunk of a prompt where activations stay in BF16
        {"name": "nvfp4_layer_t600_a16", "kind": "nvfp4_layer", "tokens": 600, "policy": "a16"},
        # a whole prompt chunk: the largest call
        {"name": "nvfp4_layer_t8192_a4", "kind": "nvfp4_layer", "tokens": 8192, "policy": "a4"},
        # eight sequences decoding at 3 bits per weight, and a prompt of 1000 tokens
        {"name": "trellis_layer_t8", "kind": "trellis_layer", "tokens": 8, "k2": 6},
        {"name": "trellis_layer_t1000", "kind": "trellis_layer", "tokens": 1000, "k2": 6},
        # the output head at 4 bits per weight, one sequence
        {"name": "trellis_head_t1", "kind": "trellis_linear", "in": HIDDEN, "out": HEAD, "tokens": 1, "k2": 8},
        # the mixture-of-experts block at 2.5 bits per weight: decoding and a prompt chunk
        {"name": "moe_block_t8", "kind": "moe_block", "hidden": 2048, "inter": 768, "experts": 512, "top_k": 10, "tokens": 8, "k2": 5},
        {"name": "moe_block_t4096", "kind": "moe_block", "hidden": 2048, "inter": 768, "experts": 512, "top_k": 10, "tokens": 4096, "k2": 5},
    ]


def _log_int(rng, low: int, high: int) -> int:
    """An integer of [low, high], spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low - 0.49), math.log(high + 0.49)))))))


def draw(rng) -> dict:
    kind = rng.choice(["nvfp4_linear", "nvfp4_layer", "nvfp4_layer", "trellis_linear", "trellis_layer", "moe_block", "moe_block"])
    if kind == "nvfp4_linear":
        if rng.random() < 0.5:
            n, k = rng.choice(LAYER_SHAPES)
        else:  # another model's width: any whole number of row tiles and scale tiles
            n, k = 128 * _log_int(rng, 4, 272), 64 * _log_int(rng, 8, 272)
        return {"kind": kind, "n": n, "k": k, "tokens": _log_int(rng, 1, 8192), "policy": rng.choice(["a16", "a4"])}
    if kind == "nvfp4_layer":
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "policy": rng.choice(["a16", "a4"])}
    if kind == "trellis_linear":
        if rng.random() < 0.3:
            out, in_, tokens = HEAD, HIDDEN, _log_int(rng, 1, 64)
        elif rng.random() < 0.5:
            (out, in_), tokens = rng.choice(LAYER_SHAPES), _log_int(rng, 1, 4096)
        else:
            out, in_, tokens = 128 * _log_int(rng, 4, 136), 128 * _log_int(rng, 4, 136), _log_int(rng, 1, 4096)
        return {"kind": kind, "in": in_, "out": out, "tokens": tokens, "k2": rng.choice(trellis.K2_VALUES)}
    if kind == "trellis_layer":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096), "k2": rng.choice(trellis.K2_VALUES)}
    hidden, inter, experts, top_k = rng.choice(MOE_GEOMETRIES)
    return {"kind": kind, "hidden": hidden, "inter": inter, "experts": experts, "top_k": top_k, "tokens": _log_int(rng, 1, 4096),
            "k2": rng.choice([4, 5, 6, 8])}


# ---- inputs ----------------------------------------------------------------------------------------

def _activations(tokens: int, width: int, gen, amp: float = 1.0) -> torch.Tensor:
    return (torch.randn(tokens, width, device="cuda", generator=gen) * amp).to(torch.bfloat16)


def _nvfp4_weight(n: int, k: int, gen) -> nvfp4.Weight:
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    natural = (torch.randn((n, k // 16), device="cuda", generator=gen).abs() + 0.1).to(torch.float8_e4m3fn).view(torch.uint8)
    stored = natural.reshape(n // 128, 4, 32, k // 64, 4).permute(0, 3, 2, 1, 4).contiguous().reshape(-1)
    return nvfp4.Weight(codes, stored, n, k, 448.0, 448.0)


def _signed(n: int, amp: float, gen) -> torch.Tensor:
    """+-(0.5 .. 2) x amp in FP16: the sign vectors of a trellis tensor."""
    v = (torch.rand(n, device="cuda", generator=gen) * 1.5 + 0.5) * amp
    return (v * (torch.randint(0, 2, (n,), device="cuda", generator=gen) * 2 - 1)).to(torch.float16)


def _trellis_weight(in_: int, out: int, k2: int, gen) -> trellis.Weight:
    words = torch.randint(-32768, 32768, ((in_ // 16) * (out // 16) * trellis.tile_words16(k2),), dtype=torch.int16, device="cuda", generator=gen)
    return trellis.Weight(words, _signed(in_, 0.05, gen), _signed(out, 0.03, gen), k2, in_, out)


def _moe_table(g: moe.Geometry, k2: int, gen) -> moe.SlotTable:
    """A layer's routed experts, every record its own random words (any bit pattern is an encoding)."""
    sizes = [moe.record_bytes(moe.PROJ_GATE_UP, k2, g), moe.record_bytes(moe.PROJ_DOWN, k2, g)]
    records = torch.randint(0, 256, (g.experts, sum(sizes)), dtype=torch.uint8, device="cuda", generator=gen)
    for at, (in_, out), (amp_in, amp_out) in ((0, (g.hidden, 2 * g.inter), (0.05, 0.03)), (sizes[0], (g.inter, g.hidden), (0.25, 0.06))):
        signs = at + in_ * out * k2 // 16
        for base, n, amp in ((signs, in_, amp_in), (signs + 2 * in_, out, amp_out)):
            records[:, base: base + 2 * n] = _signed(g.experts * n, amp, gen).view(torch.uint8).reshape(g.experts, 2 * n)
    offsets = [e * sum(sizes) + p * sizes[0] for e in range(g.experts) for p in (0, 1)]
    return moe.SlotTable.from_device_records(records.reshape(-1), offsets, [k2] * len(offsets), [(2 * e, 2 * e + 1) for e in range(g.experts)])


def _fp8_rows(rows: int, cols: int, gen) -> torch.Tensor:
    """A row-scaled E4M3 matrix as stored: codes, padding to 256 bytes, one BF16 scale per row."""
    w = torch.randn(rows, cols, device="cuda", generator=gen) * 0.02
    scale = (w.abs().amax(dim=1) / 440.0).to(torch.bfloat16)
    pad = (rows * cols + 255) // 256 * 256
    out = torch.zeros(pad + 2 * rows, dtype=torch.uint8, device="cuda")
    out[: rows * cols] = (w / scale.float().unsqueeze(1)).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8).reshape(-1)
    out[pad:] = scale.view(torch.uint8)
    return out


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, tokens = case["kind"], case["tokens"]
    s = {"kind": kind, "tokens": tokens}
    if kind in ("nvfp4_linear", "nvfp4_layer"):
        nvfp4.prepare()
        s["policy"] = POLICIES[case["policy"]]
    elif kind in ("trellis_linear", "trellis_layer"):
        trellis.prepare()
    else:
        moe.prepare()
    if kind == "nvfp4_linear":
        s["w"] = _nvfp4_weight(case["n"], case["k"], gen)
        s["x"] = _activations(tokens, case["k"], gen)
        s["ws"] = nvfp4.Workspace(nvfp4.workspace_bytes(case["n"], case["k"], s["policy"], tokens))
    elif kind == "nvfp4_layer":
        s["qkv"], s["o"] = _nvfp4_weight(sum(QKV_ROWS), HIDDEN, gen), _nvfp4_weight(HIDDEN, Q, gen)
        s["gate_up"], s["down"] = _nvfp4_weight(2 * INTER, HIDDEN, gen), _nvfp4_weight(HIDDEN, INTER, gen)
        s["x"], s["attn"], s["x_mlp"] = _activations(tokens, HIDDEN, gen), _activations(tokens, Q, gen), _activations(tokens, HIDDEN, gen)
        # one workspace for the layer, and the outputs it hands on, as an engine holds them
        s["ws"] = nvfp4.Workspace(max([nvfp4.workspace_bytes(w.n, w.k, s["policy"], tokens) for w in (s["qkv"], s["o"])] +
                                      [nvfp4.mlp_workspace_bytes(2 * INTER, HIDDEN, s["policy"], tokens)]))
        s["qkv_out"] = [torch.empty(tokens, r, dtype=torch.bfloat16, device="cuda") for r in QKV_ROWS]
        s["h"] = torch.empty(tokens, HIDDEN, dtype=torch.bfloat16, device="cuda")
    elif kind == "trellis_linear":
        s["w"] = _trellis_weight(case["in"], case["out"], case["k2"], gen)
        s["x"] = _activations(tokens, case["in"], gen)
        s["ws"] = trellis.WorkspaceBuffer(trellis.workspace_bytes(case["in"], case["out"], 1, tokens))
    elif kind == "trellis_layer":
        k2 = case["k2"]
        s["qkv"], s["o"] = [_trellis_weight(HIDDEN, r, k2, gen) for r in QKV_ROWS], _trellis_weight(Q, HIDDEN, k2, gen)
        s["gate"], s["up"], s["down"] = (_trellis_weight(i, o, k2, gen) for i, o in ((HIDDEN, INTER), (HIDDEN, INTER), (INTER, HIDDEN)))
        s["x"], s["attn"], s["x_mlp"] = _activations(tokens, HIDDEN, gen), _activations(tokens, Q, gen), _activations(tokens, HIDDEN, gen)
        s["ws"] = trellis.WorkspaceBuffer(max(trellis.workspace_bytes(i, o, c, tokens)
                                              for i, o, c in ((HIDDEN, Q, 1), (Q, HIDDEN, 1), (HIDDEN, INTER, 2), (INTER, HIDDEN, 1))))
        s["qkv_out"] = [torch.empty(tokens, r, dtype=torch.bfloat16, device="cuda") for r in QKV_ROWS]
        s["m"] = torch.empty(tokens, INTER, dtype=torch.bfloat16, device="cuda")
        s["h"] = torch.empty(tokens, HIDDEN, dtype=torch.bfloat16, device="cuda")
    elif kind == "moe_block":
        g = moe.Geometry(case["hidden"], case["inter"], case["experts"], case["top_k"])
        s["g"], s["table"] = g, _moe_table(g, case["k2"], gen)
        # the router's weights favour some experts through a channel that every token carries, so that a
        # softmax over its choices makes expert r (of a random order) popular like 1 / (r + 1)^1.1
        s["x"] = _activations(tokens, g.hidden, gen, 0.5)
        s["x"][:, 0] = 4.0
        router = torch.randn(g.experts, g.hidden, device="cuda", generator=gen) * (2.0 / math.sqrt(g.hidden))
        rank = torch.randperm(g.experts, device="cuda", generator=gen).float() + 1.0
        router[:, 0] = -ZIPF * torch.log(rank) / 4.0
        s["router"] = router.to(torch.bfloat16)
        s["shared"] = [_fp8_rows(r, c, gen) for r, c in ((g.inter, g.hidden), (g.inter, g.hidden), (g.hidden, g.inter))]
        s["gate"] = (torch.randn(g.hidden, device="cuda", generator=gen) * 0.02).to(torch.bfloat16)
        s["ws"] = moe.Workspace(min(tokens, moe.DECODE_MAX_TOKENS), tokens, geometry=g)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


# ---- one pass --------------------------------------------------------------------------------------

def run(s: dict):
    kind = s["kind"]
    if kind == "nvfp4_linear":
        return nvfp4.linear(s["x"], s["w"], policy=s["policy"], workspace=s["ws"])
    if kind == "nvfp4_layer":
        policy, ws, h = s["policy"], s["ws"], s["h"]
        q, k, v = nvfp4.linear_split(s["x"], s["qkv"], QKV_ROWS, s["qkv_out"], policy=policy, workspace=ws)
        nvfp4.linear(s["attn"], s["o"], h, policy=policy, workspace=ws)
        nvfp4.mlp(s["x_mlp"], s["gate_up"], s["down"], ws, h, policy=policy, epilogue=nvfp4.ADD)
        return [q, k, v, h]
    if kind == "trellis_linear":
        return trellis.linear(s["w"], s["x"], workspace=s["ws"])
    if kind == "trellis_layer":
        ws, h = s["ws"], s["h"]
        if s["tokens"] <= trellis.DECODE_MAX_TOKENS:
            q, k, v = trellis.linear_group(s["qkv"], s["x"], s["qkv_out"])
        else:  # the grouped call has no workspace: wide calls go one by one
            q, k, v = (trellis.linear(w, s["x"], y, workspace=ws) for w, y in zip(s["qkv"], s["qkv_out"]))
        trellis.linear(s["o"], s["attn"], h, workspace=ws)
        m = trellis.linear_swiglu(s["gate"], s["up"], s["x_mlp"], s["m"], workspace=ws)
        trellis.linear(s["down"], m, h, epilogue=trellis.ADD, workspace=ws)
        return [q, k, v, h]
    x, g, ws = s["x"], s["g"], s["ws"]
    ids, weights, _ = moe.router(x, s["router"], g)
    experts = moe.experts_decode if s["tokens"] <= moe.DECODE_MAX_TOKENS else moe.experts_prefill
    experts(x, ids, weights, s["table"], ws)
    shared, _ = moe.shared_expert(*s["shared"], x, g)
    return moe.combine(ws, shared, x, s["gate"])


# ---- what a pass cannot do without ---------------------------------------------------------------

def _hit_experts(case: dict) -> float:
    """Experts that a call's tokens choose at all, in expectation (choices drawn one by one)."""
    p = [(r + 1.0) ** -ZIPF for r in range(case["experts"])]
    total, choices = sum(p), case["tokens"] * case["top_k"]
    return sum(1.0 - (1.0 - v / total) ** choices for v in p)


def work(case: dict) -> dict:
    kind, t = case["kind"], case["tokens"]
    if kind == "nvfp4_linear":
        n, k = case["n"], case["k"]
        return {"bytes": n * k * 9 // 16 + 2 * t * (n + k), "flops": 2.0 * t * n * k}
    if kind == "trellis_linear":
        i, o = case["in"], case["out"]
        return {"bytes": i * o * case["k2"] // 16 + 2 * (i + o) + 2 * t * (i + o), "flops": 2.0 * t * i * o}
    if kind in ("nvfp4_layer", "trellis_layer"):
        bits16 = 9 if kind == "nvfp4_layer" else case["k2"]
        return {"bytes": DENSE_PARAMS * bits16 // 16 + 2 * t * (2 * HIDDEN + Q + sum(QKV_ROWS) + HIDDEN), "flops": 2.0 * t * DENSE_PARAMS}
    hidden, inter, experts = case["hidden"], case["inter"], case["experts"]
    expert = 3 * hidden * inter
    weights = _hit_experts(case) * expert * case["k2"] / 16 + expert + 2 * experts * hidden
    return {"bytes": weights + 2 * t * 2 * hidden, "flops": 2.0 * t * (expert * (case["top_k"] + 1) + experts * hidden)}


def tolerance(case: dict) -> dict:
    if case["kind"] == "moe_block":
        # BF16 output; where two experts tie at the router's last choice, the order of its sums decides between them
        return {"rel": 1e-2, "max": 0.5}
    if case["kind"] == "nvfp4_linear":
        return {"rel": 4e-3}   # FP32 sums, rounded once to BF16
    return {"rel": 1e-2}       # a layer: BF16 (or FP4) between its two MLP products
