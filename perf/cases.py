"""The work that this framework is timed on: what a serving engine has it do, through the entry points an engine calls.

Five kinds of case, each a dict of plain values:

  linear   one call of the `linear` operator (runtime.ops) from eager code, as an engine's linear layer makes it: 1 row to
           prefill-sized batches, one matrix or a fused group, padded input widths and trimmed output columns
  stack    the linears of a few dense layers as a captured decode step (runtime.layerset.DecodeLayerSet.replay)
  step     a full decode step with attention, norms and the residual stream, captured (runtime.decode_step.DecodeStep.replay)
  moe      one routed-expert layer (kernels.base.B200Backend.run_moe on a caller-owned workspace), eager as in a prefill or
           replayed from a CUDA graph as in a decode step
  load     a checkpoint's fused group brought into the resident layout (kernels.linear.prepare), once per module at start-up

Sizes: the 27B-shape layer (hidden 5120, q 5120, kv 1024, ffn 17408), the 256-expert layer (hidden 2048, intermediate 512,
top-8), the 4096 x 4096 matrix and the small matrix of the smoke run, and generic sizes between them.  Inputs are N(0, 1)
activations, uniform trellis bits, random signs with per-channel scales, softmax routing over random logits.
"""
from __future__ import annotations

import math

import torch

from trellis_serve_b200.kernels import linear as lin
from trellis_serve_b200.kernels import moe
from trellis_serve_b200.kernels.base import B200Backend
from trellis_serve_b200.runtime import ops
from trellis_serve_b200.runtime.decode_step import DecodeStep, ModelShape
from trellis_serve_b200.runtime.layerset import DecodeLayerSet, LayerShape

DEV = torch.device("cuda:0")
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}
MCG, MUL1, THREE_INST = 1, 2, 0


# ---------------------------------------------------------------------------------------------------------------- cases

def _linear(name, rows, k, widths, K, codebook, dtype, pad=0, trim=0):
    """widths: output columns of the group's matrices, e.g. "5120,1024,1024"; pad: columns by which the activations are
    narrower than the stored input width; trim: true output columns of the last matrix are that many fewer than stored."""
    return {"name": name, "kind": "linear", "rows": rows, "k": k, "widths": widths, "K": K, "codebook": codebook, "dtype": dtype,
            "pad": pad, "trim": trim}


def listed():
    return [
        # The smallest call: a draft or adapter-sized matrix, one token.  Launch and host time are all of it.
        _linear("linear_1row_1024x640", 1, 1024, "640", 3, THREE_INST, "f16"),
        # One token through a mid-sized matrix.
        _linear("linear_1row_4096x4096", 1, 4096, "4096", 4, THREE_INST, "f16"),
        # A few concurrent sequences (or draft tokens being verified) through a fused group in bf16, the engines' default.
        _linear("linear_5rows_qkv_27b", 5, 5120, "5120,1024,1024", 3, MCG, "bf16"),
        # The largest decode batch one pass over the weights serves, at a high bit rate with the third codebook.
        _linear("linear_16rows_down_27b", 16, 17408, "5120", 6, MUL1, "f16"),
        # A short prompt with a ragged row count through a matrix whose true sizes are not the stored, padded ones.
        _linear("linear_57rows_ragged", 57, 5120, "5120", 4, MCG, "bf16", pad=56, trim=40),
        # A prefill chunk through the largest group of the 27B-shape layer: the case with the most arithmetic.
        _linear("linear_2048rows_gate_up_27b", 2048, 5120, "17408,17408", 4, MCG, "f16"),
        # All linears of eight 27B-shape layers for one token, as captured by an engine (990 MB of weights).
        {"name": "stack_8layers_27b", "kind": "stack", "layers": 8, "rows": 1, "K": 3, "codebook": THREE_INST, "dtype": "f16",
         "hidden": 5120, "q_out": 5120, "kv_out": 1024, "ffn": 17408},
        # One token through eight layers with attention over a 2048-token cache.
        {"name": "step_8layers_27b", "kind": "step", "layers": 8, "rows": 1, "K": 3, "codebook": THREE_INST, "dtype": "f16",
         "hidden": 5120, "q_heads": 40, "kv_heads": 8, "ffn": 17408, "context": 2048},
        # Routed experts: one decoded token, a decode batch (both captured), and a prefill chunk (eager).
        {"name": "moe_1token", "kind": "moe", "tokens": 1, "hidden": 2048, "inter": 512, "experts": 256, "top_k": 8, "K": 3, "more": 0,
         "codebook": THREE_INST, "dtype": "bf16", "graph": True},
        {"name": "moe_64tokens", "kind": "moe", "tokens": 64, "hidden": 2048, "inter": 512, "experts": 256, "top_k": 8, "K": 3, "more": 0,
         "codebook": THREE_INST, "dtype": "bf16", "graph": True},
        {"name": "moe_2048tokens", "kind": "moe", "tokens": 2048, "hidden": 2048, "inter": 512, "experts": 256, "top_k": 8, "K": 3,
         "more": 0, "codebook": THREE_INST, "dtype": "bf16", "graph": False},
        # Start-up: the gate|up group of one 27B-shape layer from the stored to the resident layout.
        {"name": "load_gate_up_27b", "kind": "load", "k": 5120, "widths": "17408,17408", "K": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log128(rng, lo, hi):
    return 128 * max(1, _log(rng, lo / 128, hi / 128))


def _widths(rng, k):
    """One matrix, a pair (gate|up) or three (q|k|v), at most 180 M weights in all."""
    cap = 180_000_000 // k
    shards = rng.choice([1, 1, 2, 3])
    if shards == 1:
        w = [_log128(rng, 512, 17408)]
    elif shards == 2:
        w = [_log128(rng, 512, 17408)] * 2
    else:
        w = [_log128(rng, 1024, 5120)] + [_log128(rng, 256, 1024)] * 2
    w = [max(128, min(n, cap // len(w) // 128 * 128)) for n in w]
    return ",".join(str(n) for n in w)


def draw(rng):
    K, codebook, dtype = rng.randint(2, 8), rng.choice([0, 0, 1, 1, 2]), rng.choice(["f16", "bf16"])
    kind = rng.choice(["linear", "linear", "linear", "linear", "many", "many", "stack", "step", "moe", "moe", "moe", "load"])
    if kind in ("linear", "many"):
        k = _log128(rng, 1024, 17408)
        rows = rng.randint(1, 16) if kind == "linear" else _log(rng, 17, 2048)
        pad = rng.randrange(8, 121, 8) if rng.random() < 0.25 else 0
        trim = rng.randrange(8, 121, 8) if rng.random() < 0.25 else 0
        c = _linear("", rows, k, _widths(rng, k), K, codebook, dtype, pad, trim)
    elif kind == "stack":
        c = {"kind": "stack", "layers": rng.randint(2, 8), "rows": rng.choice([1, 1, 2, rng.randint(3, 16)]), "K": rng.randint(2, 6),
             "codebook": codebook, "dtype": dtype, "hidden": _log128(rng, 1024, 5120), "q_out": _log128(rng, 1024, 5120),
             "kv_out": 128 * rng.randint(1, 8), "ffn": _log128(rng, 2048, 17408)}
    elif kind == "step":
        kv = rng.choice([1, 2, 4, 8])
        c = {"kind": "step", "layers": rng.randint(2, 8), "rows": rng.choice([1, 1, 2, rng.randint(3, 8)]), "K": rng.randint(2, 6),
             "codebook": codebook, "dtype": dtype, "hidden": _log128(rng, 1024, 5120), "q_heads": kv * rng.randint(8 // kv, min(8, 40 // kv)),
             "kv_heads": kv, "ffn": _log128(rng, 2048, 17408), "context": _log(rng, 64, 4096)}
    elif kind == "moe":
        tokens = _log(rng, 1, 2048)
        experts = rng.choice([32, 64, 128, 256])
        c = {"kind": "moe", "tokens": tokens, "hidden": rng.choice([1024, 1536, 2048]), "inter": rng.choice([384, 512, 768]),
             "experts": experts, "top_k": rng.choice([2, 4, 6, 8]), "K": rng.randint(2, 5), "more": rng.choice([0, 0, 0, experts // 4]),
             "codebook": codebook, "dtype": dtype, "graph": tokens <= 128 and rng.random() < 0.7}
    else:
        k = _log128(rng, 1024, 17408)
        c = {"kind": "load", "k": k, "widths": _widths(rng, k), "K": K}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _trellis(g, k, n, K, *lead):
    return torch.randint(-32768, 32768, (*lead, k // 16, n // 16, 16 * K), dtype=torch.int16, device=DEV, generator=g)


def _scales(g, magnitude, *shape):
    """Sign vectors with per-channel scales around `magnitude`."""
    s = torch.randint(0, 2, shape, device=DEV, generator=g, dtype=torch.int32) * 2 - 1
    return (s * magnitude * (1.0 + 0.1 * torch.randn(shape, device=DEV, generator=g))).to(torch.float16)


def _normal(g, dtype, *shape):
    return torch.randn(shape, device=DEV, generator=g).to(DTYPES[dtype])


def _out_scale(k):
    """Real svh vectors carry the 1 / sqrt(k) of the product (codebook values have a deviation of about 1.24)."""
    return 1.0 / (1.2437 * math.sqrt(k))


def _group(g, k, widths, K):
    widths = [int(n) for n in widths.split(",")]
    return ([_trellis(g, k, n, K) for n in widths], [_scales(g, 1.0, k) for _ in widths], [_scales(g, _out_scale(k), n) for n in widths])


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "load":
        trellis, suh, svh = _group(g, case["k"], case["widths"], case["K"])
        return {"kind": kind, "trellis": trellis, "suh": suh, "svh": svh}
    if kind == "linear":
        widths = [int(n) for n in case["widths"].split(",")]
        packed, suh, svh, ends = lin.prepare(*_group(g, case["k"], case["widths"], case["K"]))
        return {"kind": kind, "x": _normal(g, case["dtype"], case["rows"], case["k"] - case["pad"]), "weights": [packed, suh, svh],
                "ends": ends, "codebooks": [case["codebook"]] * len(widths), "widths": widths[:-1] + [widths[-1] - case["trim"]]}
    if kind == "stack":
        s = DecodeLayerSet(case["layers"], case["K"], case["codebook"], case["rows"],
                           LayerShape(case["hidden"], case["q_out"], case["kv_out"], case["ffn"]), seed=seed, device=DEV, dtype=DTYPES[case["dtype"]])
        for layer in s.groups:
            for group in layer:
                group.svh.mul_(_out_scale(group.packed.shape[1] * 128))
        for x in (s.x_hidden, s.x_attn, s.x_ffn):
            x.copy_(_normal(g, case["dtype"], *x.shape))
        s.capture()
        return {"kind": kind, "stack": s}
    if kind == "step":
        shape = ModelShape(case["hidden"], case["q_heads"], case["kv_heads"], 128, case["ffn"], case["layers"])
        s = DecodeStep(shape, case["K"], case["codebook"], case["context"], case["rows"], device=DEV, dtype=DTYPES[case["dtype"]], seed=seed)
        s.h_in.copy_(_normal(g, case["dtype"], *s.h_in.shape))
        s.capture()
        return {"kind": kind, "step": s}
    h, i, e = case["hidden"], case["inter"], case["experts"]

    def experts(k, n):
        """The first e - more experts at K bits, the last `more` at K + 1."""
        few = e - case["more"]
        t = list(_trellis(g, k, n, case["K"], few)) + (list(_trellis(g, k, n, case["K"] + 1, case["more"])) if case["more"] else [])
        return t, list(_scales(g, 1.0, e, k)), list(_scales(g, _out_scale(k), e, n))

    pack = moe.prepare_mixed(experts(h, i), experts(h, i), experts(i, h), case["codebook"])
    tokens, top_k = case["tokens"], case["top_k"]
    logits = torch.randn((tokens, e), device=DEV, generator=g)
    weights, ids = torch.topk(torch.softmax(logits, dim=1), top_k, dim=1)
    weights, ids = (weights / weights.sum(dim=1, keepdim=True)).contiguous(), ids.to(torch.int32).contiguous()
    x = _normal(g, case["dtype"], tokens, h)
    out = torch.empty_like(x)
    need = moe.layer_workspace_bytes([p.num_experts for p in pack.packs], h, i, case["codebook"], tokens, top_k)
    workspace = torch.zeros(need, dtype=torch.uint8, device=DEV)
    backend = B200Backend()
    state = {"kind": kind, "args": (pack, x, ids, weights, out, workspace, None), "backend": backend, "out": out, "graph": None}
    if case["graph"]:
        backend.run_moe(*state["args"])
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            backend.run_moe(*state["args"])
        state["graph"] = graph
    return state


# ---------------------------------------------------------------------------------------------------------------- a pass

def run(state):
    kind = state["kind"]
    if kind == "linear":
        return ops.linear(state["x"], [], [], [], [], [], 0, state["weights"], state["ends"], state["codebooks"], state["widths"])
    if kind == "stack":
        s = state["stack"]
        s.replay()
        return [s.y_qkv, s.y_o, s.y_gu, s.y_down]
    if kind == "step":
        s = state["step"]
        return {"hidden": s.replay(), "cache": s.kv}
    if kind == "moe":
        if state["graph"] is not None:
            state["graph"].replay()
        else:
            state["backend"].run_moe(*state["args"])
        return state["out"]
    packed, suh, svh, ends = lin.prepare(state["trellis"], state["suh"], state["svh"])
    return {"packed": packed, "suh": suh, "svh": svh, "ends": ends}


# ---------------------------------------------------------------------------------------------------------------- figures

def _linear_work(rows, k, n, shards, K):
    """Weights, activations and outputs once, sign vectors; the product (the rotations are a few percent of it at most)."""
    return k * n * K / 8 + 2.0 * rows * (k + n) + 2.0 * (shards * k + n), 2.0 * rows * k * n


def work(case):
    kind = case["kind"]
    if kind == "load":
        weights = case["k"] * sum(int(n) for n in case["widths"].split(","))
        return {"bytes": 2 * weights * case["K"] / 8, "flops": 0}
    if kind == "linear":
        widths = [int(n) for n in case["widths"].split(",")]
        b, f = _linear_work(case["rows"], case["k"], sum(widths), len(widths), case["K"])
        return {"bytes": b, "flops": f}
    if kind in ("stack", "step"):
        h, ffn, rows, K = case["hidden"], case["ffn"], case["rows"], case["K"]
        q, kv = (case["q_out"], case["kv_out"]) if kind == "stack" else (case["q_heads"] * 128, case["kv_heads"] * 128)
        parts = [_linear_work(rows, k, n, s, K) for k, n, s in ((h, q + 2 * kv, 3), (q, h, 1), (h, 2 * ffn, 2), (ffn, h, 1))]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
        if kind == "step":
            b += 2 * rows * case["kv_heads"] * 128 * case["context"] * 2
            f += 4.0 * rows * case["q_heads"] * 128 * case["context"]
        return {"bytes": case["layers"] * b, "flops": case["layers"] * f}
    h, i, e, t, top_k = (case[n] for n in ("hidden", "inter", "experts", "tokens", "top_k"))
    touched = e * (1.0 - (1.0 - top_k / e) ** t)            # experts that t tokens are expected to reach
    bits = case["K"] + case["more"] / e
    return {"bytes": touched * (3 * h * i * bits / 8 + 2 * (3 * h + 3 * i)) + 4.0 * t * h, "flops": 6.0 * t * top_k * h * i}


def tolerance(case):
    kind = case["kind"]
    if kind == "load":
        return "exact"                                       # a permutation of the stored bits
    bf16 = case["dtype"] == "bf16"
    if kind in ("linear", "stack"):
        # fp32 sums in another order, fp16 rounding of the rotated product and of the result; bf16 results can differ by
        # one unit in the last place, 2^-8 of a value.
        return {"rel": 6e-3, "max": 0.03} if bf16 else {"rel": 2e-3, "max": 0.01}
    if kind == "moe":                                        # two products with fp16 values between them
        return {"rel": 8e-3, "max": 0.05} if bf16 else {"rel": 4e-3, "max": 0.02}
    # Up to eight layers one behind the other, each rounding the stream and its activations to 16 bits.
    return {"rel": 2e-2, "max": 0.2} if bf16 else {"rel": 6e-3, "max": 0.06}
