"""The performance cases of libkq: the work its users have it do, called the way they call it.

A host program keeps one context (`acquire_gpu`), uploads packed weights once, and then, per
token or per request, replays a recorded decoder step, runs a prompt through the layers, or
calls single quantized linears.  `listed()` are the cases that are always timed, `draw()` gives
further ones of the same ranges, `prepare()` builds what such a program holds before the call,
and `run()` is the call.

Weights have the distributions of the reference's quantiser on normal weights: int4 nibbles
uniform over 0..15 with scales |N(0, 0.02)| / 7, int8 uniform over -127..127 with scales
|N(0, 0.02)| / 127; activations are N(0, 1).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import karume_b200 as kb

# The two decoders whose projections are measured: (hidden, q, kv, ffn, vocabulary, tied head).
# "8b" is the Llama-8B-shaped decoder of bench_workload.py, "1.5b" the 1.5B-class one whose
# LM head is also its embedding table.
DECODERS = {
    "8b": dict(hidden=4096, q=4096, kv=1024, ffn=14336, vocab=128256, tied=False),
    "1.5b": dict(hidden=1536, q=1536, kv=256, ffn=8960, vocab=151936, tied=True),
}
EPS = 1e-5
MAX_WORK = 2048 * 4096 * 14336  # m * n * k of the largest single linear
TORCH_DTYPE = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # One token of one conversation: the step every chat user waits for, latency above all.
        dict(name="decode_8b_1row", kind="decode", model="8b", layers=32, rows=1, scale="f16"),
        # A pipeline stage (8 layers and the head) that serves sixteen conversations at once.
        dict(name="decode_8b_16rows", kind="decode", model="8b", layers=8, rows=16, scale="f16"),
        # A small decoder on a handful of rows: a few users, or the tokens of one speculative draft.
        dict(name="decode_1.5b_4rows", kind="decode", model="1.5b", layers=12, rows=4, scale="f32"),
        # A prompt through the first layers and the head: f32 activations and f32 scales, as the
        # reference computes and ships them; prompts have any length.
        dict(name="prefill_1.5b_333rows", kind="prefill", model="1.5b", layers=4, rows=333, scale="f32"),
        # The smallest call: one projection of one token, where launch and host path count.
        dict(name="linear_i4_m1", kind="linear", storage="i4", group=32, scale="f16", x="f32", m=1, k=4096, n=4096),
        # The LM head of one token over an int8 vocabulary: the largest matrix a token reads.
        dict(name="linear_i8_head_m1", kind="linear", storage="i8", group=0, scale="f16", x="f32", m=1, k=1536, n=151936),
        # Verifying a speculative draft of eight tokens with binary16 activations.
        dict(name="linear_i4_f16_m8", kind="linear", storage="i4", group=32, scale="f16", x="f16", m=8, k=4096, n=11008),
        # The up projection of a long prompt in bf16: the largest contraction.
        dict(name="linear_i4_bf16_m2048", kind="linear", storage="i4", group=32, scale="f16", x="bf16", m=2048, k=4096, n=14336),
        # A prompt over int8 weights with the reference's f32 activations, of no round length.
        dict(name="linear_i8_m257", kind="linear", storage="i8", group=0, scale="f32", x="f32", m=257, k=1536, n=8960),
        # An embedding model's projection, exported with groups of sixteen for accuracy.
        dict(name="linear_i4_g16_m65", kind="linear", storage="i4", group=16, scale="f32", x="f32", m=65, k=1152, n=3072),
        # Integer-dot layers of an image transformer: every token of a latent at once, int8 weights ...
        dict(name="a8_i8_m4096", kind="a8", storage="i8", group=0, scale="f32", m=4096, k=2048, n=8192),
        # ... and int4 weights on a smaller latent.
        dict(name="a8_i4_m1000", kind="a8", storage="i4", group=32, scale="f32", m=1000, k=2048, n=2048),
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of lo..hi."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["decode", "prefill", "linear", "a8"], [4, 2, 10, 4])[0]
    scale = rng.choice(["f16", "f32"])
    if kind == "decode":
        return dict(kind=kind, model=rng.choice(["8b", "1.5b"]), layers=_spread(rng, 1, 16), rows=rng.choice([1, 1, rng.randint(2, 16)]),
                    scale=scale)
    if kind == "prefill":
        return dict(kind=kind, model=rng.choice(["8b", "1.5b"]), layers=rng.randint(1, 4), rows=_spread(rng, 17, 1024), scale=scale)
    storage = rng.choice(["i4", "i4", "i8"])
    group = rng.choice([32, 32, 32, 32, 16, 64, 128]) if storage == "i4" else 0
    step = max(64, group)  # int4 rows are whole groups; projections are multiples of 64 wide
    if kind == "a8":
        m, x = _spread(rng, 1, 4096), None
    else:
        m = rng.choice([1, rng.randint(2, 16), _spread(rng, 17, 2048)])
        x = rng.choice(["f32", "f32", "f16", "bf16"])
    while True:
        k = step * max(1, round(_spread(rng, 256, 14336) / step))
        n = _spread(rng, 64, 65536 if m <= 16 else 14336)
        if rng.random() < 0.75:
            n = 16 * max(1, round(n / 16))  # the others are ragged
        if m * n * k <= MAX_WORK and n * k <= 2 ** 28:
            break
    case = dict(kind=kind, storage=storage, group=group, scale=scale, m=m, k=k, n=n)
    if x:
        case["x"] = x
    return case


# ---- what a user's program holds -----------------------------------------------------------

_gpu_kept = None


def _gpu():
    """The process's one context, on a stream of its own that torch uses too."""
    global _gpu_kept
    if _gpu_kept is None:
        torch.cuda.set_stream(torch.cuda.Stream())
        _gpu_kept = kb.acquire_gpu(0)
    return _gpu_kept


class _State:
    """Resident weights, buffers and a recorded step; gives its device memory back when dropped."""

    def __init__(self, case):
        self.case, self.gpu = case, _gpu()
        self.weights, self.plan, self.graph = {}, None, None

    def __del__(self):
        if self.plan is not None:
            self.gpu.plan_free(self.plan)
        if self.graph is not None:
            self.gpu.graph_free(self.graph)
        for w in self.weights.values():
            w.free()


class _Packed:
    """Packed weights drawn from one seeded pool; every matrix starts somewhere else in it."""

    def __init__(self, seed, storage, group, scale, largest):
        self.rng = np.random.default_rng([seed, 17])
        self.storage, self.group = storage, group
        numel = largest + (1 << 16)
        if storage == "i4":
            self.pool = self.rng.integers(0, 256, numel // 2, dtype=np.uint8)
            spread, scales = 0.02 / 7, numel // group
        else:
            self.pool = self.rng.integers(-127, 128, numel, dtype=np.int8)
            spread, scales = 0.02 / 127, 1 << 18
        s = np.abs(self.rng.standard_normal(scales, dtype=np.float32)) * np.float32(spread)
        s = np.maximum(s, np.float32(1e-7)).astype(np.float16)
        self.scales = s if scale == "f16" else s.astype(np.float32)

    def _cut(self, pool, count):
        at = 16 * int(self.rng.integers(0, (pool.size - count) // 16 + 1))
        return pool[at:at + count]

    def upload(self, gpu, n, k):
        if self.storage == "i4":
            payload, scale = self._cut(self.pool, n * k // 2), self._cut(self.scales, n * (k // self.group))
        else:
            payload, scale = self._cut(self.pool, n * k), self._cut(self.scales, n)
        return gpu.upload_weight(self.storage, payload, scale, (n, k), self.group)


def _matmuls(case):
    """(name, n, k) of every weight of a decoder case."""
    d = DECODERS[case["model"]]
    out = []
    for i in range(case["layers"]):
        out += [(f"{i}.q", d["q"], d["hidden"]), (f"{i}.k", d["kv"], d["hidden"]), (f"{i}.v", d["kv"], d["hidden"]),
                (f"{i}.o", d["hidden"], d["q"]), (f"{i}.gate", d["ffn"], d["hidden"]), (f"{i}.up", d["ffn"], d["hidden"]),
                (f"{i}.down", d["hidden"], d["ffn"])]
    return out + [("head", d["vocab"], d["hidden"])]


def prepare(case, seed):
    s = _State(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    if case["kind"] in ("linear", "a8"):
        packed = _Packed(seed, case["storage"], case["group"], case["scale"], case["n"] * case["k"])
        s.weights["w"] = packed.upload(s.gpu, case["n"], case["k"])
        s.x = normal(case["m"], case["k"])
        if case["kind"] == "linear":
            s.x = s.x.to(TORCH_DTYPE[case["x"]])
        s.bias = normal(case["n"])
    else:
        _prepare_decoder(s, case, seed, normal, gen)
    torch.cuda.current_stream().synchronize()
    return s


def _prepare_decoder(s, case, seed, normal, gen):
    d, rows = DECODERS[case["model"]], case["rows"]
    shapes = _matmuls(case)
    packed = _Packed(seed, "i4", 32, case["scale"], max(n * k for _, n, k in shapes))
    for name, n, k in shapes:
        s.weights[name] = packed.upload(s.gpu, n, k)
    s.norms = 1.0 + 0.1 * normal(2 * case["layers"] + 1, d["hidden"])
    s.biases = {name: 0.02 * normal(n) for name, n, _ in shapes}
    s.ids = torch.randint(d["vocab"], (rows,), generator=gen, device="cuda", dtype=torch.int32)
    s.x = normal(rows, d["hidden"])  # the token rows; a tied table's rows replace them in run()
    s.query = torch.empty(rows, d["q"], device="cuda")
    s.cache = torch.empty(case["layers"], 2, rows, d["kv"], device="cuda")  # this step's keys and values
    s.act = torch.empty(rows, d["ffn"], device="cuda")
    s.hidden = torch.empty(rows, d["hidden"], device="cuda")
    s.logits = torch.empty(1 if case["kind"] == "prefill" else rows, d["vocab"], device="cuda")
    if case["kind"] == "decode":
        _record(s)


def _enqueue_layers(s):
    """The matmuls of the layers with their norms, gates and residuals (attention is the host's:
    o takes q)."""
    g, w, b = s.gpu, s.weights, s.biases
    cur = s.x
    for i in range(s.case["layers"]):
        names = [f"{i}.q", f"{i}.k", f"{i}.v"]
        g.linear_fused(cur, [w[t] for t in names], [b[t] for t in names], [s.query, s.cache[i, 0], s.cache[i, 1]],
                       norm_weight=s.norms[2 * i], eps=EPS)
        g.linear_fused(s.query, [w[f"{i}.o"]], [b[f"{i}.o"]], [s.hidden], residual=cur)
        cur = s.hidden
        names = [f"{i}.gate", f"{i}.up"]
        g.linear_fused(cur, [w[t] for t in names], [b[t] for t in names], [s.act], norm_weight=s.norms[2 * i + 1], eps=EPS,
                       swiglu=True)
        g.linear_fused(s.act, [w[f"{i}.down"]], [b[f"{i}.down"]], [s.hidden], residual=cur)
    return cur


def _enqueue_head(s, rows):
    s.gpu.linear_fused(rows, [s.weights["head"]], [s.biases["head"]], [s.logits], norm_weight=s.norms[-1], eps=EPS)


def _record(s):
    """One replayable step: a fused plan where the library has one for these rows, else a graph."""
    g = s.gpu
    try:
        g.plan_begin()
        _enqueue_head(s, _enqueue_layers(s))
        s.plan = g.plan_end()
    except kb.KqError as e:
        if e.status != "KQ_ERR_UNSUPPORTED":
            raise
        _enqueue_head(s, _enqueue_layers(s))  # the context's scratch grows before a capture, not in it
        g.sync()
        g.graph_begin()
        _enqueue_head(s, _enqueue_layers(s))
        s.graph = g.graph_end()


# ---- the calls ---------------------------------------------------------------------------------

def run(s):
    case, g = s.case, s.gpu
    if case["kind"] == "linear":
        return g.linear(s.x, s.weights["w"], s.bias)
    if case["kind"] == "a8":
        q, scale = g.quantize_rows(s.x)
        return {"q": q, "scale": scale, "out": g.linear_a8(q, scale, s.weights["w"], s.bias)}
    if DECODERS[case["model"]]["tied"]:
        g.embedding(s.ids, s.weights["head"], out=s.x)
    if case["kind"] == "prefill":
        h = _enqueue_layers(s)
        _enqueue_head(s, h[-1:])
    elif s.plan is not None:
        g.plan_launch(s.plan)
    else:
        g.graph_launch(s.graph)
    return {"cache": s.cache, "hidden": s.hidden, "logits": s.logits}


# ---- what a call cannot do without -----------------------------------------------------------

def _weight_bytes(storage, group, scale, n, k):
    each = 2 if scale == "f16" else 4
    return n * k // 2 + n * (k // group) * each if storage == "i4" else n * k + n * each


def work(case):
    if case["kind"] in ("linear", "a8"):
        m, n, k = case["m"], case["n"], case["k"]
        held = _weight_bytes(case["storage"], case["group"], case["scale"], n, k)
        x_each = 4 if case.get("x", "f32") == "f32" else 2
        q = m * k + 4 * m if case["kind"] == "a8" else 0
        return {"bytes": held + x_each * m * k + q + 4 * n + 4 * m * n, "flops": 2 * m * n * k}
    d, rows = DECODERS[case["model"]], case["rows"]
    total = flops = 0
    for name, n, k in _matmuls(case):
        m = 1 if name == "head" and case["kind"] == "prefill" else rows
        total += _weight_bytes("i4", 32, case["scale"], n, k) + 4 * n
        flops += 2 * m * n * k
    total += 4 * d["hidden"] * (2 * case["layers"] + 1)                       # norm weights
    total += 4 * rows * (2 * d["hidden"] + 2 * d["kv"] * case["layers"])     # token rows in, hidden rows and cache out
    total += 4 * d["vocab"] * (1 if case["kind"] == "prefill" else rows)      # logits
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["kind"] == "a8":
        return "exact"  # integer sums, and a fixed order of the few f32 operations
    if case.get("x") == "bf16" and case["m"] > 16:
        return {"rel": 5e-3}  # weights rounded to bf16
    if case["kind"] == "prefill":
        return {"rel": 1e-4}  # a chain of f32 layers whose operands are carried as two 16-bit numbers each
    if case["kind"] == "linear" and case["m"] > 16:
        return {"rel": 3e-5}
    return {"rel": 1e-5}
