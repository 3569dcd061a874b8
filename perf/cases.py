"""The work that a program built on this library has it do, as timed cases: `listed()` names them, `draw()` gives more of the
same ranges, `prepare()` makes what a program holds before the call (weights, plans, activations), `run()` is one pass through
the public entry points of ijah_b200.engine, `work()` the bytes and operations a pass cannot do without, `tolerance()` how far
another correct implementation at the same precision may be off.

Weights and activations are the synthetic ones of ijah_b200.synth and of the model object (uniform trellis words, signs +-1,
scales |N(0, 1)| * 0.02, router N(0, 0.02), activations N(0, 1) rounded to f16). Sizes are those of bench.py and of the tests.
"""
import math

import numpy as np
import torch

from ijah_b200 import engine as E
from ijah_b200 import synth

HIDDEN, INTER, EXPERTS, TOPK = 2048, 768, 512, 10  # the MoE block of bench.py; every eighth drawn block has another one's
OTHER = (2560, 640)                                # the reference's hidden and intermediate sizes
VOCAB = 151936

_eng = None


def engine():
    global _eng
    if _eng is None:
        _eng = E.Engine()
    return _eng


def listed():
    return [
        # one Linear for one row: an expert-sized matrix, nothing but latency
        {"name": "linear_1row", "op": "linear", "n_in": 2048, "n_out": 768, "k": 5, "rows": 1},
        # the attention projections of a layer (q, k, v on shared rows, then o) in token-by-token decode
        {"name": "trunk_1row", "op": "trunk", "hidden": 2048, "q_out": 4096, "kv_out": 512, "k": 6, "rows": 1},
        # the same at 8 bits for a ragged batch of sequences
        {"name": "trunk_27rows", "op": "trunk", "hidden": 2048, "q_out": 4096, "kv_out": 512, "k": 8, "rows": 27},
        # one MoE block: token-by-token decode, the verify width of a speculative round, the widest decode batch
        {"name": "block_1row", "op": "block", "hidden": HIDDEN, "inter": INTER, "k": 5, "rows": 1},
        {"name": "block_6rows", "op": "block", "hidden": HIDDEN, "inter": INTER, "k": 5, "rows": 6},
        {"name": "block_64rows", "op": "block", "hidden": HIDDEN, "inter": INTER, "k": 5, "rows": 64},
        # prompt prefill of one MoE block: a short ragged prompt with even routing (every expert touched, few rows each) and
        # a full chunk whose routing follows a Zipf law (a few experts get most rows)
        {"name": "prefill_333", "op": "prefill", "hidden": HIDDEN, "inter": INTER, "k": 5, "tokens": 333, "zipf": False},
        {"name": "prefill_4096", "op": "prefill", "hidden": HIDDEN, "inter": INTER, "k": 5, "tokens": 4096, "zipf": True},
        # prompt prefill of an attention projection, ragged
        {"name": "linear_1000rows", "op": "linear_prefill", "n_in": 2048, "n_out": 4096, "k": 6, "rows": 1000},
        # the 8-bit affine LM head at the reference's size for a verify round
        {"name": "head_q8_4rows", "op": "q8", "n_in": 2560, "n_out": 248320, "group": 64, "rows": 4},
        # whole decode steps with host tokens in and logits out: a batch of two sequences with four verify tokens each, and a
        # prompt that goes through the stack in chunks of 32 rows
        {"name": "stack_8rows", "op": "stack", "layers": 4, "rows": 8},
        {"name": "stack_prompt_100", "op": "prompt", "layers": 2, "chunk": 32, "tokens": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["linear", "linear", "trunk", "block", "block", "block", "prefill", "prefill", "linear_prefill", "q8", "stack", "prompt"])
    if op == "linear":
        return {"op": op, "n_in": 64 * _log(rng, 8, 64), "n_out": 64 * _log(rng, 8, 64), "k": rng.randint(4, 8), "rows": _log(rng, 1, 64)}
    if op == "trunk":
        return {"op": op, "hidden": 256 * _log(rng, 4, 12), "q_out": 512 * _log(rng, 2, 8), "kv_out": 256 * rng.randint(1, 4), "k": rng.randint(4, 8),
                "rows": _log(rng, 1, 64)}
    if op in ("block", "prefill"):
        h, i = (HIDDEN, INTER) if rng.random() < 0.875 or op == "prefill" else OTHER
        c = {"op": op, "hidden": h, "inter": i, "k": rng.choice([4, 5, 5, 5, 6])}
        if op == "block":
            c["rows"] = _log(rng, 1, 64)
        else:
            c.update(tokens=_log(rng, 65, 4000), zipf=rng.random() < 0.5)
        return c
    if op == "linear_prefill":
        return {"op": op, "n_in": 128 * _log(rng, 8, 32), "n_out": 256 * _log(rng, 2, 16), "k": rng.randint(4, 8), "rows": _log(rng, 65, 4000)}
    if op == "q8":
        return {"op": op, "n_in": 256 * rng.randint(4, 10), "n_out": _log(rng, 2048, 240000), "group": rng.choice([64, 128]), "rows": _log(rng, 1, 16)}
    if op == "stack":
        return {"op": op, "layers": rng.randint(1, 4), "rows": _log(rng, 1, 16)}
    return {"op": op, "layers": rng.randint(1, 3), "chunk": rng.choice([16, 32, 64]), "tokens": _log(rng, 20, 130)}


class Freed:
    """Holds a handle of the library and releases it with the state."""

    def __init__(self, handle):
        self.h = handle

    def __del__(self):
        torch.cuda.synchronize()
        self.h.free()


def _rows(gen, rows, n):
    return torch.randn((rows, n), device="cuda", generator=gen).to(torch.float16).to(torch.float32)


def _exl3(gen, n_in, n_out, k):
    tr = torch.randint(-32768, 32768, (n_in // 16, n_out // 16, 16 * k), dtype=torch.int16, device="cuda", generator=gen)
    suh = (torch.randint(0, 2, (n_in,), device="cuda", generator=gen) * 2 - 1).to(torch.float16)
    sign = (torch.randint(0, 2, (n_out,), device="cuda", generator=gen) * 2 - 1).to(torch.float32)
    svh = (sign * torch.randn((n_out,), device="cuda", generator=gen).abs() * 0.02).to(torch.float16)
    return E.Exl3Linear.from_device(engine(), tr, suh, svh)


def _q8(gen, c):
    n_in, n_out, group = c["n_in"], c["n_out"], c["group"]
    lin = E.Q8Linear.__new__(E.Q8Linear)  # (the constructor takes host arrays; these are made on the device)
    lin.eng, lin.n_in, lin.n_out, lin.group = engine(), n_in, n_out, group
    w = torch.empty((n_out, n_in), dtype=torch.uint8, device="cuda")
    for o in range(0, n_out, 16384):  # N(128, 32) as trained tables have it, in pieces that bound the temporaries
        w[o:o + 16384] = (torch.randn((min(16384, n_out - o), n_in), device="cuda", generator=gen) * 32 + 128).round().clamp(0, 255).to(torch.uint8)
    std = 0.02
    sc = (std / 32) * (1 + 0.1 * torch.randn((n_out, n_in // group), device="cuda", generator=gen))
    bi = -128 * sc + 0.1 * std * torch.randn((n_out, n_in // group), device="cuda", generator=gen)
    lin.t = (w, sc.to(torch.bfloat16), bi.to(torch.bfloat16))
    lin.c = E.Q8WeightC(lin.t[0].data_ptr(), lin.t[1].data_ptr(), lin.t[2].data_ptr(), n_in, n_out, group)
    return lin


def _stack_desc(layers):
    return dict(layers=layers, hidden=HIDDEN, inter=INTER, experts=EXPERTS, top_k=TOPK, k_expert=5, k_shared=6, q_out=4096, kv_out=512, heads=16,
                kv_heads=2, head_dim=256, k_trunk=6, k_trunk_alt=8, alt_every=4, vocab=VOCAB, kv_positions=8192, expert_first=0, expert_count=0,
                ep_world=1)


def prepare(case, seed):
    op = case["op"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if op in ("linear", "linear_prefill"):
        return {"op": op, "lin": _exl3(gen, case["n_in"], case["n_out"], case["k"]), "x": _rows(gen, case["rows"], case["n_in"])}
    if op == "trunk":
        h, q, kv, r = case["hidden"], case["q_out"], case["kv_out"], case["rows"]
        qkv = [_exl3(gen, h, n, case["k"]) for n in (q, kv, kv)]
        return {"op": op, "qkv": qkv, "o": _exl3(gen, q, h, case["k"]), "x": _rows(gen, r, h), "att": _rows(gen, r, q)}
    if op in ("block", "prefill"):
        t = synth.moe_layer(seed, hidden=case["hidden"], inter=case["inter"], experts=EXPERTS, k_expert=case["k"], k_shared=6)
        n = case["rows"] if op == "block" else case["tokens"]
        x = _rows(gen, n, case["hidden"])
        if case.get("zipf"):
            synth.zipf_router_bias(t)
            x[:, 0] = 1.0
        return {"op": op, "blk": Freed(E.MoeBlock(engine(), t, top_k=TOPK, max_rows=n if op == "block" else 16)), "x": x}
    if op == "q8":
        return {"op": op, "lin": _q8(gen, case), "x": _rows(gen, case["rows"], case["n_in"])}
    rows = case["rows"] if op == "stack" else case["tokens"]
    m = engine().fn_model(desc=_stack_desc(case["layers"]), seed=seed, max_rows=case["rows"] if op == "stack" else case["chunk"])
    tokens = np.random.default_rng(seed).integers(0, VOCAB, rows).astype(np.int32)
    s = {"op": op, "model": Freed(m), "tokens": tokens}
    run(dict(s, tokens=(tokens + 1) % VOCAB))  # a serving program has warmed its step up before the first request
    return s


def run(state):
    op = state["op"]
    if op == "linear":
        return state["lin"](state["x"])
    if op == "trunk":
        x = state["x"]
        outs = [torch.empty((x.shape[0], l.n_out), dtype=torch.float32, device="cuda") for l in state["qkv"]]
        E.linear_multi(engine(), state["qkv"], x, outs)
        return (*outs, state["o"](state["att"]))
    if op == "block":
        return state["blk"].h.forward(state["x"])
    if op == "prefill":
        return state["blk"].h.prefill(state["x"])
    if op == "linear_prefill":
        return state["lin"].prefill(state["x"])
    if op == "q8":
        return state["lin"](state["x"])
    # the logits come back to the host (the greedy tokens, their argmax, with them)
    if op == "stack":
        return state["model"].h.step_rows(state["tokens"], want_logits=True)[1]
    return state["model"].h.prefill(state["tokens"])[1]


def _exl3_bytes(n_in, n_out, k):
    return n_in * n_out * k / 8 + 2 * n_in + 2 * n_out


def _distinct(rows):
    return EXPERTS * (1 - (1 - TOPK / EXPERTS) ** rows)  # expected number of experts that `rows` rows touch


def _block_work(h, i, k, rows):
    b = EXPERTS * h * 2 + h * 2 + 2 * _exl3_bytes(h, i, 6) + _exl3_bytes(i, h, 6)
    b += _distinct(rows) * (2 * _exl3_bytes(h, i, k) + _exl3_bytes(i, h, k)) + 2 * rows * h * 4
    return b, rows * ((TOPK + 1) * 6 * h * i + 2 * h * EXPERTS)


def _stack_work(layers, rows, logit_rows):
    q, kv = 4096, 512
    bb, bf = _block_work(HIDDEN, INTER, 5, rows)
    per = bb + _exl3_bytes(HIDDEN, q, 6) + 2 * _exl3_bytes(HIDDEN, kv, 6) + _exl3_bytes(q, HIDDEN, 6) + 2 * 8192 * kv * 2
    perf = bf + 2 * rows * (2 * HIDDEN * q + 2 * HIDDEN * kv) + 4 * rows * 8192 * q
    head = (VOCAB * HIDDEN * 2 + logit_rows * VOCAB * 4) if logit_rows else 0
    return layers * per + head, layers * perf + 2 * logit_rows * VOCAB * HIDDEN


def work(case):
    op = case["op"]
    if op in ("linear", "linear_prefill"):
        n, m, r = case["n_in"], case["n_out"], case["rows"]
        return {"bytes": _exl3_bytes(n, m, case["k"]) + 4 * r * (n + m), "flops": 2 * r * n * m}
    if op == "trunk":
        h, q, kv, k, r = (case[x] for x in ("hidden", "q_out", "kv_out", "k", "rows"))
        b = _exl3_bytes(h, q, k) + 2 * _exl3_bytes(h, kv, k) + _exl3_bytes(q, h, k) + 4 * r * (2 * h + 2 * q + 2 * kv)
        return {"bytes": b, "flops": 2 * r * (2 * h * q + 2 * h * kv)}
    if op in ("block", "prefill"):
        b, f = _block_work(case["hidden"], case["inter"], case["k"], case["rows"] if op == "block" else case["tokens"])
        return {"bytes": b, "flops": f}
    if op == "q8":
        n, m, r = case["n_in"], case["n_out"], case["rows"]
        return {"bytes": n * m + 4 * n * m / case["group"] + 4 * r * (n + m), "flops": 2 * r * n * m}
    if op == "stack":
        b, f = _stack_work(case["layers"], case["rows"], case["rows"])
        return {"bytes": b, "flops": f}
    n, c, b, f = case["tokens"], case["chunk"], 0, 0
    for at in range(0, n, c):  # every chunk streams the experts it touches; the head runs for the prompt's last rows
        r = min(c, n - at)
        bb, ff = _stack_work(case["layers"], r, 1 if at + c >= n else 0)
        b, f = b + bb, f + ff
    return {"bytes": b, "flops": f}


def tolerance(case):
    # Measured against products in f64 with the Hadamard transforms as matrix products (linears, q8), between the decode and
    # the prefill kernels (blocks), and between one step of 8 rows and the same rows alone, in threes and in fours (stacks):
    # each bound is about four times the largest difference seen.
    op = case["op"]
    if op in ("linear", "linear_prefill", "trunk"):
        return {"rel": 2.5e-5, "max": 2e-3}  # f32 sums; an operand now and then rounds to the neighbouring f16 value: 6e-6, 4e-4
    if op in ("block", "prefill"):
        return {"rel": 2e-4, "max": 8e-3}  # the same twice in a row: 5e-5, 1.6e-3
    if op == "q8":
        return {"rel": 1e-6, "max": 1e-5}  # f32 throughout: 2.4e-7, 1.3e-6
    # Four layers of that and a bf16 rounding in front of the head: 8.6e-4, 4.2e-3. In 3 of 40 batches of 8 rows one row's
    # tenth and eleventh expert were so close that the summation order decided: 0.015 over the batch, that row's logits 0.04.
    return {"rel": 0.025, "max": 0.4}
